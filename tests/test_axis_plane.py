"""x and y line passes of small square grids in one launch (a plane of one field per CTA): the
same stages in the same order as the separate launches, which pass timing keeps, so the fields
must agree bit for bit; the launch count shows which form ran.  Sizes: every compiled length,
both sides of the rule's plane counts (64 and 72 points: two planes per SM, FP32 at most four),
the crystal on three fields and the free-space return on two."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu


def run(n, nt, precision, timing, nrt=3):
    cfg = co.make_config(nx=n, ny=n, nt=nt, nz=4, n_steps=4, LX=300.0, LY=300.0, Lcr=3000.0, P=400.0, w0=40.0, FWHM=3.0,
                         t_window=25.0, pump_mode="focused-pulsed", Rs=0.9, total_rt=nrt, precision=precision)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.init_fields(cfg, 31, 0.02, idler_copy=True)
    sim.set_pass_timing(timing)
    before = sim.kernel_launches
    sim.run_round_trips(nrt)
    sim.synchronize()
    launches = sim.kernel_launches - before
    out = [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
    steps = params.n_steps
    sim.close()
    return out, launches, steps


def one_launch(n, precision, planes):
    if n <= 48:
        return True
    if precision == co.FP64:
        return n <= 72 and planes >= 296
    return n <= 64 and 296 <= planes <= 592


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("n,nt", [(16, 32), (24, 12), (32, 64), (36, 36), (48, 96), (64, 96), (64, 108), (64, 144),
                                  (64, 192), (64, 216), (72, 96), (72, 128)])
def test_one_launch_equals_two(n, nt, precision):
    a, la, steps = run(n, nt, precision, True)
    b, lb, _ = run(n, nt, precision, False)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    saved = 3 * steps * one_launch(n, precision, 3 * nt) + 2 * one_launch(n, precision, 2 * nt)
    assert la - lb == saved

"""A batch's round-trip graph against its resident instances: a batch that has drained takes
instances with another number of z-steps on the same grid (nothing else about the launches
changes), fewer and more, plain and corrected physics (phase tables per z-step)."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu

TUNING = {k: dict(threads=128, tile=1024, r1=4) for k in "txy"}


def config(nx, ny, nt, precision=co.FP64, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=5, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", total_rt=9, precision=precision)
    kw.update(over)
    return co.make_config(**kw)


def standalone(cfg, nrt, seed):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.set_tuning(TUNING)
    sim.set_plane_pass(0)
    sim.init_fields(cfg, seed, 0.02, idler_copy=True)
    sim.run_round_trips(nrt)
    out = [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
    sim.close()
    return out


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("over", [{}, dict(flags=co.DISPERSION | co.DIFFRACTION | co.PHYSICS, Lambda=6.5)])
def test_drained_batch_takes_another_step_count(precision, over):
    b = co.Batch(precision, 2, 1 << 30, tuning=TUNING)
    for k, steps in enumerate([6, 3, 3, 9]):
        cfg = config(16, 16, 32, precision, nz=steps + 1, n_steps=steps, **over)
        s = b.add(cfg)
        b.init_fields(s, cfg, 20 + k, 0.02, idler_copy=True)
        b.run_round_trips(2)
        for a, c in zip([b.get_field(s, f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)], standalone(cfg, 2, 20 + k)):
            assert np.array_equal(a, c), steps
        b.remove(s)
    b.close()

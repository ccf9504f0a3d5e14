"""Line-specialised x- and y-passes: compiled bodies for the axis lengths of LENGTHS, one field
per tile, run in place of the generic tiles under every classic x / y setting.  Round trips
(crystal steps, free-space return) must match the FP64 oracle within the form's tolerance
(FP32 1e-5, FP64 1e-10) for every length on either axis, on ragged last tiles (line counts
that are no multiple of a tile's), on square grids (the y-pass's compiled row stride) and
beside axes without a body; a batch's slots equal standalone solvers bit for bit."""
import numpy as np
import pytest

import cuopo3d_b200 as co
from golden_cases import rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

TOL = {co.FP32: 1e-5, co.FP64: 1e-10}
LENGTHS = [16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 384, 512]
TUNING = {k: dict(threads=128, tile=1024, r1=4) for k in "txy"}


def config(nx, ny, nt, precision, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=4, LX=300.0, LY=250.0, Lcr=3000.0, P=400.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", gdd_gamma=0.6, Rs=0.9, total_rt=3)
    kw.update(over)
    return kw, co.make_config(precision=precision, **kw)


def standalone(cfg, tuning=None, nrt=2, seed=31):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    if tuning:
        sim.set_tuning(tuning)
        sim.set_plane_pass(0)
    sim.init_fields(cfg, seed, 0.02, idler_copy=True)
    sim.run_round_trips(nrt)
    out = [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
    sim.close()
    return out


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("n", LENGTHS)
def test_every_length_vs_oracle(n, precision):
    # x of length n (36 rows x 9 planes: ragged row tiles), y of length n beside a generic
    # x axis (12 columns: a ragged column tile), and the square grid
    grids = [(n, 36, 12), (12, n, 8)] + ([(n, n, 8)] if n <= 144 else [])
    for grid in grids:
        kw, cfg = config(*grid, precision)
        st = po.Setup(po.make_phys(**kw))
        api = st.api_complex()
        s0 = co.noise(31, 0.02, api.size).reshape(api.shape)
        ref = po.round_trips(st, api, api, s0, s0, 2)
        for a, b in zip(standalone(cfg, TUNING), ref):
            assert rel_l2(a, b) < TOL[precision], (grid, rel_l2(a, b))


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_batch_equals_standalone(precision):
    grids = [(16, 96, 16), (72, 72, 16), (128, 32, 16), (12, 48, 16), (256, 16, 16)]
    b = co.Batch(precision, len(grids), 8 << 30, tuning=TUNING)
    slots = []
    for k, g in enumerate(grids):
        _, cfg = config(*g, precision, P=100.0 + 50 * k)
        s = b.add(cfg)
        b.init_fields(s, cfg, 31 + k, 0.02, idler_copy=True)
        slots.append((s, cfg))
        b.run_round_trips(1 if k == 2 else 0)  # groups join after the graph was built
    b.run_round_trips(2)
    for k, (s, cfg) in enumerate(slots):
        nrt = 3 if k <= 2 else 2
        for a, c in zip([b.get_field(s, f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)],
                        standalone(cfg, TUNING, nrt, 31 + k)):
            assert np.array_equal(a, c), grids[k]
    b.close()

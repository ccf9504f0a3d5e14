"""Line t-pass bodies of the time axes in LENGTHS (two- and three-stage plans), which replace the
generic t-pass under every classic setting: round trips with GDD, mirrors and, in turn,
the EOM or the corrected physics match the FP64 oracle within the form's tolerance (FP32
1e-5, FP64 1e-10); planes that hold no whole tile keep the generic body; a batch's slots
(bodies, the line setting's own axes and the generic body mixed) equal standalone solvers
bit for bit."""
import numpy as np
import pytest

import cuopo3d_b200 as co
from golden_cases import rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

TOL = {co.FP32: 1e-5, co.FP64: 1e-10}
LENGTHS = [32, 36, 48, 72, 96, 108, 144, 192, 216, 288, 384, 432, 512, 576, 768, 864, 1024]
TUNING = {"t": dict(threads=128, tile=1024, r1=4), "x": dict(threads=128, tile=1024, r1=4),
          "y": dict(threads=128, tile=1024, r1=4)}


def config(nx, ny, nt, precision, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=4, LX=300.0, LY=250.0, Lcr=3000.0, P=400.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", gdd_gamma=0.6, Rs=0.9, total_rt=3)
    kw.update(over)
    return kw, co.make_config(precision=precision, **kw)


def standalone(cfg, tuning, nrt, seed):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.set_tuning(tuning)
    sim.set_plane_pass(0)
    sim.init_fields(cfg, seed, 0.02, idler_copy=True)
    sim.run_round_trips(nrt)
    out = [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
    sim.close()
    return out


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("nt", LENGTHS)
def test_every_length_vs_oracle(nt, precision):
    overs = [dict(eom_beta=0.4, eom_fpm=0.05),
             dict(flags=co.DISPERSION | co.DIFFRACTION | co.PHYSICS, Lambda=6.5)]
    # whole tiles on a ragged row (12 pixels), and a plane of 9 rows of 6 (no whole tile)
    for k, (nx, ny) in enumerate([(12, 8), (8, 8), (6, 9) if nt <= 216 else (12, 8)]):
        kw, cfg = config(nx, ny, nt, precision, **overs[k % 2])
        flags = kw.pop("flags", co.DISPERSION | co.DIFFRACTION)
        if nx == 6:
            flags = co.DISPERSION  # 6 and 9 points are no diffraction axes
            cfg = co.make_config(precision=precision, flags=flags, **kw)
        st = po.Setup(po.make_phys(flags=flags, **kw))
        api = st.api_complex()
        s0 = co.noise(31, 0.02, api.size).reshape(api.shape)
        ref = po.round_trips(st, api, api, s0, s0, 2)
        for a, b in zip(standalone(cfg, TUNING, 2, 31), ref):
            assert rel_l2(a, b) < TOL[precision], ((nx, ny, nt), rel_l2(a, b))


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("line", [0, co.LINE])
def test_batch_equals_standalone(precision, line):
    grids = [(16, 16, 96), (16, 16, 128), (24, 16, 1024), (12, 16, 64), (16, 8, 24), (16, 16, 512), (16, 24, 216)]
    tun = {**TUNING, "t": dict(threads=128, tile=1024, r1=4 + line)}
    b = co.Batch(precision, len(grids), 8 << 30, tuning=tun)
    slots = []
    for k, g in enumerate(grids):
        over = dict(flags=co.DISPERSION | co.DIFFRACTION | co.PHYSICS, Lambda=6.5) if k % 3 == 2 else {}
        _, cfg = config(*g, precision, P=100.0 + 50 * k, **over)
        s = b.add(cfg)
        b.init_fields(s, cfg, 31 + k, 0.02, idler_copy=True)
        slots.append((s, cfg))
        if k == 2:
            b.run_round_trips(1)  # other groups join after the graph was built
    b.run_round_trips(2)
    for k, (s, cfg) in enumerate(slots):
        for a, c in zip([b.get_field(s, f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)],
                        standalone(cfg, tun, 3 if k <= 2 else 2, 31 + k)):
            assert np.array_equal(a, c), grids[k]
    b.close()

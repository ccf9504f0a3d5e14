"""The plane-wave (1 x 1) solver's whole-crystal kernel on clusters of 1, 4, 8 and 16 CTAs
(untuned and autotuned solvers): single passes and round trips with EOM, GDD, mirrors and,
in turn, the corrected physics, against the FP64 oracle within the form's tolerance (FP32
1e-5, FP64 1e-10); and a solver's repeated single passes (launched directly the first time,
as a graph after it), 1-D and 3-D, bit for bit the same."""
import numpy as np
import pytest

import cuopo3d_b200 as co
from golden_cases import rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

TOL = {co.FP32: 1e-5, co.FP64: 1e-10}


def setup(precision, **over):
    kw = dict(nx=1, ny=1, nt=256, nz=8, LX=1.0, LY=1.0, Lcr=10000.0, P=2.0, w0=40.0, FWHM=1.0, t_window=20.0,
              pump_mode="waveplane-pulsed", gdd_gamma=0.8, Rs=0.95, total_rt=4, flags=co.DISPERSION)
    kw.update(over)
    cfg = co.make_config(precision=precision, **kw)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    st = po.Setup(po.make_phys(**kw))
    api = st.api_complex()
    s0 = co.noise(3, 1e-3, api.size).reshape(api.shape)
    return co.Simulation(params, w), st, api, s0


def upload(sim, api, s0):
    for which, arr in ((co.FIELD_API, api), (co.FIELD_AP, api), (co.FIELD_AS, s0), (co.FIELD_AI, s0)):
        sim.set_field(which, arr)


def fields(sim):
    return [sim.get_field(f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("nt", [16, 36, 108, 288, 576, 1024, 2304, 4096])
def test_round_trips_vs_oracle(nt, precision):
    for over in (dict(eom_beta=0.6, eom_fpm=0.05),
                 dict(flags=co.DISPERSION | co.PHYSICS, Lambda=6.5),
                 dict(flags=0, gdd_gamma=0.0)):
        sim, st, api, s0 = setup(precision, nt=nt, **over)
        if nt == 576:
            sim.autotune()
        upload(sim, api, s0)
        sim.run_round_trips(3)
        ref = po.round_trips(st, api, api, s0, s0, 3)
        for a, b in zip(fields(sim), ref):
            assert rel_l2(a, b) < TOL[precision], (over, rel_l2(a, b))


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("grid", [(1, 1, 1152), (1, 1, 108), (16, 24, 48)])
def test_repeated_single_passes(grid, precision):
    over = dict(zip(("nx", "ny", "nt"), grid))
    if grid[0] > 1:
        over.update(LX=300.0, LY=250.0, flags=co.DISPERSION | co.DIFFRACTION)
    sim, st, api, s0 = setup(precision, **over)
    runs = []
    for _ in range(3):
        upload(sim, api, s0)
        sim.run_single_pass()
        runs.append(fields(sim))
    for r in runs[1:]:
        for a, b in zip(runs[0], r):
            assert np.array_equal(a, b)
    for a, b in zip(runs[0], po.single_pass(st, api, s0, s0)):
        assert rel_l2(a, b) < TOL[precision]

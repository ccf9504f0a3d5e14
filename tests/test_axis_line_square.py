"""x- and y-line passes on planes of many tiles: square grids of the longer compiled lengths (the y kernels
with a compiled row stride, and the TMA-fed bodies with many column boxes a plane) and long y axes
beside 36 columns (whole tiles and a ragged one), round trips against the FP64 oracle within the
forms' tolerances (FP32 1e-5, FP64 1e-10)."""
import pytest

import cuopo3d_b200 as co
from golden_cases import rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

TOL = {co.FP32: 1e-5, co.FP64: 1e-10}


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("nx,ny", [(192, 192), (216, 216), (256, 256), (384, 384), (512, 512), (36, 128), (36, 192),
                                   (36, 256), (36, 512)])
def test_many_tiles_vs_oracle(nx, ny, precision):
    kw = dict(nx=nx, ny=ny, nt=8, nz=3, LX=300.0, LY=250.0, Lcr=3000.0, P=400.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", gdd_gamma=0.6, Rs=0.9, total_rt=3)
    cfg = co.make_config(precision=precision, **kw)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.set_plane_pass(0)
    sim.init_fields(cfg, 31, 0.02, idler_copy=True)
    sim.run_round_trips(2)
    st = po.Setup(po.make_phys(**kw))
    api = st.api_complex()
    s0 = co.noise(31, 0.02, api.size).reshape(api.shape)
    ref = po.round_trips(st, api, api, s0, s0, 2)
    for f, b in zip((co.FIELD_AP, co.FIELD_AS, co.FIELD_AI), ref):
        a = sim.get_field(f)
        assert rel_l2(a, b) < TOL[precision], rel_l2(a, b)
    sim.close()

"""The bounded tile waits of the TMA-fed x- and y-passes (line bodies from 128 points on) under
opo_set_wait_limit: with a bound of a few clock cycles a pass gives up its wait (the tile's copy
takes far longer) and ends; the host gets OPO_ERR_CUDA at its next synchronisation, the
fields count as lost until all four are uploaded, and with the default bound restored the
same solver gives the same bits as one that never timed out."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("nx,ny", [(128, 12), (16, 192), (256, 256)])
def test_wait_expiry_is_reported_and_the_solver_recovers(nx, ny, precision):
    cfg = co.make_config(nx=nx, ny=ny, nt=16, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=400.0, w0=40.0, FWHM=3.0,
                         t_window=25.0, pump_mode="focused-pulsed", total_rt=50, precision=precision)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)

    def run(sim):
        api = co.pump_field(cfg)
        s0 = co.noise(8, 0.02, api.size).reshape(api.shape)
        for which, arr in ((co.FIELD_API, api), (co.FIELD_AP, api), (co.FIELD_AS, s0), (co.FIELD_AI, s0)):
            sim.set_field(which, arr)
        sim.run_round_trips(2)
        return [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]

    fresh = co.Simulation(params, w)
    fresh.set_plane_pass(0)  # 12 points have no body: the default is a plane pass there
    want = run(fresh)
    fresh.close()
    sim = co.Simulation(params, w)
    sim.set_plane_pass(0)
    run(sim)  # graphs captured with the default bound
    sim.synchronize()
    sim.set_wait_limit(4)
    sim.run_round_trips(1)
    with pytest.raises(co.OpoError) as e:
        sim.synchronize()
    assert e.value.code == co.OPO_ERR_CUDA and "x- or y-pass" in str(e.value) and "timed out" in str(e.value)
    for call in (lambda: sim.get_field(co.FIELD_AS), sim.run_single_pass, sim.field_sums):
        with pytest.raises(co.OpoError) as e:
            call()
        assert e.value.code == co.OPO_ERR_CUDA and "lost" in str(e.value)
    sim.set_wait_limit(0)
    for a, b in zip(run(sim), want):
        assert np.array_equal(a, b)
    sim.close()

"""An allocation that fails is reported by the call that made it and by no later one: another solver runs
on (the generic kernels check their launches through the runtime's last error)."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu


def config(nx, ny, nt, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", total_rt=9, precision=co.FP64)
    kw.update(over)
    return co.make_config(**kw)


def solver(cfg):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    return co.Simulation(params, w)


def test_another_solver_runs_on():
    cfg = config(12, 12, 24)  # no compiled bodies
    sim = solver(cfg)
    sim.set_plane_pass(0)
    runs = []
    for k in range(2):
        sim.init_fields(cfg, 5, 0.02, idler_copy=True)
        if k:
            with pytest.raises(co.OpoError):
                hold = [solver(config(1024, 1024, 1728)) for _ in range(2)]  # 116 GB each
                del hold
        sim.run_single_pass()
        runs.append(sim.get_field(co.FIELD_AS))
    assert np.array_equal(*runs)
    sim.close()

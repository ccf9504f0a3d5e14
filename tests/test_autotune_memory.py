"""opo_autotune where every pass has a compiled body: there is nothing to time, so it allocates no scratch
fields (a device whose memory has no room for them does not fail it), and the passes it leaves
work on the solver's own fields."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_no_scratch_where_every_pass_has_a_body(precision):
    import torch
    cfg = co.make_config(nx=128, ny=192, nt=432, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0,
                         t_window=25.0, pump_mode="focused-pulsed", total_rt=9, precision=precision)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)

    def fields(tune):
        sim = co.Simulation(params, w)
        sim.init_fields(cfg, 5, 0.02, idler_copy=True)
        sim.run_round_trips(1)
        sim.synchronize()
        if tune:
            scratch = 4 * 128 * 192 * 432 * (16 if precision == co.FP64 else 8)
            hold = []
            while torch.cuda.mem_get_info()[0] > scratch // 2:
                room = torch.cuda.mem_get_info()[0] - scratch // 4
                hold.append(torch.empty(min(room, 32 << 30), dtype=torch.uint8, device="cuda"))
            sim.autotune()
            del hold
            torch.cuda.empty_cache()
        sim.run_round_trips(1)
        out = [sim.get_field(f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
        sim.close()
        return out

    for a, b in zip(fields(False), fields(True)):
        assert np.array_equal(a, b)

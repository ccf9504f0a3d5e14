"""opo_autotune where every pass has a compiled body: there is nothing to time, so it allocates no scratch
fields (a device whose memory has no room for them does not fail it), and the passes it leaves
work on the solver's own fields."""
import ctypes

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


class Hold:
    """All device memory but about `leave` bytes."""

    def __init__(self, leave):
        import torch
        self.cu, self.held = ctypes.CDLL("libcuda.so.1"), []
        for unit in (8 << 30, 64 << 20, 2 << 20):
            while torch.cuda.mem_get_info()[0] >= leave + unit:
                p = ctypes.c_ulonglong()
                if self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(unit)):
                    break
                self.held.append(p)

    def release(self):
        for p in self.held:
            self.cu.cuMemFree_v2(p)
        self.held = []


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_autotune_that_runs_out_of_memory_leaves_a_working_solver(precision):
    """Room for the scratch fields but hardly for the candidates' kernels and tables: whatever opo_autotune
    answers, the passes then work on the solver's own fields (the y line body reads them
    through tensor maps)."""
    nx, ny, nt = 288, 128, 24  # t and x are timed, y has a TMA-fed body
    cfg = co.make_config(nx=nx, ny=ny, nt=nt, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0,
                         t_window=25.0, pump_mode="focused-pulsed", total_rt=9, precision=precision)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    scratch = 4 * nx * ny * nt * (16 if precision == co.FP64 else 8)
    for leave in (0, 2 << 20, 6 << 20, 20 << 20):
        outs = []
        for tune in (False, True):
            sim = co.Simulation(params, w)
            sim.set_plane_pass(0)
            sim.init_fields(cfg, 5, 0.02, idler_copy=True)
            sim.run_round_trips(1)
            sim.synchronize()
            if tune:
                hold = Hold(scratch + leave)
                try:
                    sim.autotune()
                except co.OpoError as e:
                    print("leaving", leave, e)
                finally:
                    hold.release()
            sim.run_round_trips(1)
            outs.append([sim.get_field(f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)])
            sim.close()
        for a, b in zip(*outs):
            assert np.linalg.norm(a - b) < (1e-10 if precision == co.FP64 else 1e-5) * np.linalg.norm(a)

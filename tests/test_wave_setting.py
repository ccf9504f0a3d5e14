"""Settings of the plane-wave (1 x 1) solver: under a t-pass setting that names the line form, a
standalone solver and a batch's slot run the same t-pass, bit for bit; the solver's own setting
(the plane-wave kernel) survives get_tuning -> set_tuning, and a batch accepts it."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu


def config(nt, precision):
    return co.make_config(nx=1, ny=1, nt=nt, nz=8, LX=1.0, LY=1.0, Lcr=10000.0, P=2.0, w0=40.0, FWHM=1.0, t_window=20.0,
                          pump_mode="waveplane-pulsed", gdd_gamma=0.8, Rs=0.95, total_rt=20, flags=co.DISPERSION,
                          precision=precision)


def solver(cfg):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    return co.Simulation(params, w)


def run(sim, cfg):
    sim.init_fields(cfg, 3, 1e-3, idler_copy=True)
    sim.run_round_trips(2)
    return [sim.get_field(f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("nt", [64, 96, 256, 1024])
def test_line_setting_equals_a_batch_slot(nt, precision):
    cfg = config(nt, precision)
    tun = {"t": dict(threads=128, tile=2048, r1=4 + co.LINE), "x": dict(threads=128, tile=2048, r1=8),
           "y": dict(threads=128, tile=2048, r1=8)}
    sim = solver(cfg)
    sim.set_tuning(tun)
    alone = run(sim, cfg)
    sim.close()
    b = co.Batch(precision, 1, 1 << 30, tuning=tun)
    s = b.add(cfg)
    b.init_fields(s, cfg, 3, 1e-3, idler_copy=True)
    b.run_round_trips(2)
    for f, a in zip((co.FIELD_AP, co.FIELD_AS, co.FIELD_AI), alone):
        assert np.array_equal(b.get_field(s, f), a)
    b.close()


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_own_setting_is_kept(precision):
    cfg = config(256, precision)
    sim = solver(cfg)
    own = run(sim, cfg)
    tun = sim.tuning
    assert tun["t"]["r1"] & co.WAVE
    sim.close()
    for tuned in (False, True):
        sim = solver(cfg)
        if tuned:
            sim.autotune()
        else:
            sim.set_tuning({k: dict(threads=128, tile=2048, r1=8) for k in "txy"})
            sim.set_tuning(tun)
        for a, b in zip(run(sim, cfg), own):
            assert np.array_equal(a, b)
        n = sim.kernel_launches
        sim.run_round_trips(1)
        assert sim.kernel_launches == n + 1
        sim.close()
    b = co.Batch(precision, 1, 1 << 30, tuning=tun)
    s = b.add(cfg)
    b.init_fields(s, cfg, 3, 1e-3, idler_copy=True)
    b.run_round_trips(1)
    b.close()

"""Configuration calls while the caller captures the solver's or the batch's stream (relaxed mode): what
they upload is there for the launches that follow, and does not become part of the caller's
graph."""
import ctypes

import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu

TUNING = {k: dict(threads=128, tile=1024, r1=4) for k in "txy"}
RELAXED = 2


class Capture:
    def __init__(self, stream):
        self.cu, self.stream, self.graph = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(stream), ctypes.c_void_p()

    def __enter__(self):
        assert self.cu.cuStreamBeginCapture_v2(self.stream, RELAXED) == 0
        return self

    def __exit__(self, *exc):
        assert self.cu.cuStreamEndCapture(self.stream, ctypes.byref(self.graph)) == 0
        n = ctypes.c_size_t(0)
        assert self.cu.cuGraphGetNodes(self.graph, None, ctypes.byref(n)) == 0
        self.nodes = n.value
        assert self.cu.cuGraphDestroy(self.graph) == 0


def setup(precision):
    cfg = co.make_config(nx=16, ny=24, nt=32, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0,
                         t_window=25.0, pump_mode="focused-pulsed", total_rt=9, precision=precision)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.set_plane_pass(0)
    sim.init_fields(cfg, 5, 0.02, idler_copy=True)
    sim.synchronize()
    return cfg, sim


def fields(sim):
    return [sim.get_field(f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_set_tuning_under_capture(precision):
    _, a = setup(precision)
    a.set_tuning(TUNING)
    a.run_single_pass()
    _, b = setup(precision)
    with Capture(b.stream) as c:
        for _ in range(4):  # past the first configuration's own table area
            b.set_tuning(TUNING)
    assert c.nodes == 0
    b.run_single_pass()
    for x, y in zip(fields(a), fields(b)):
        assert np.array_equal(x, y)
    a.close()
    b.close()


def test_batch_add_under_capture():
    cfg, a = setup(co.FP64)
    a.set_tuning(TUNING)
    a.run_round_trips(1)
    b = co.Batch(co.FP64, 1, 1 << 30, tuning=TUNING)
    with Capture(b.stream) as c:
        s = b.add(cfg)
    assert c.nodes == 0
    b.init_fields(s, cfg, 5, 0.02, idler_copy=True)
    b.run_round_trips(1)
    for f, x in zip((co.FIELD_AP, co.FIELD_AS, co.FIELD_AI), fields(a)):
        assert np.array_equal(b.get_field(s, f), x)
    a.close()
    b.close()

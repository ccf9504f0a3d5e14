"""A batch's round-trip graph against its resident instances: a batch that has drained takes
instances with another number of z-steps on the same grid (nothing else about the launches
changes), fewer and more, plain and corrected physics (phase tables per z-step)."""
import numpy as np
import pytest

import cuopo3d_b200 as co

pytestmark = pytest.mark.gpu

TUNING = {k: dict(threads=128, tile=1024, r1=4) for k in "txy"}


def config(nx, ny, nt, precision=co.FP64, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=5, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", total_rt=9, precision=precision)
    kw.update(over)
    return co.make_config(**kw)


def standalone(cfg, nrt, seed):
    params, _ = co.derive(cfg)
    _, w = co.time_freq(cfg.nt, params.t_window)
    sim = co.Simulation(params, w)
    sim.set_tuning(TUNING)
    sim.set_plane_pass(0)
    sim.init_fields(cfg, seed, 0.02, idler_copy=True)
    sim.run_round_trips(nrt)
    out = [sim.get_field(k) for k in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]
    sim.close()
    return out


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
@pytest.mark.parametrize("over", [{}, dict(flags=co.DISPERSION | co.DIFFRACTION | co.PHYSICS, Lambda=6.5)])
def test_drained_batch_takes_another_step_count(precision, over):
    b = co.Batch(precision, 2, 1 << 30, tuning=TUNING)
    for k, steps in enumerate([6, 3, 3, 9]):
        cfg = config(16, 16, 32, precision, nz=steps + 1, n_steps=steps, **over)
        s = b.add(cfg)
        b.init_fields(s, cfg, 20 + k, 0.02, idler_copy=True)
        b.run_round_trips(2)
        for a, c in zip([b.get_field(s, f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)], standalone(cfg, 2, 20 + k)):
            assert np.array_equal(a, c), steps
        b.remove(s)
    b.close()


def fields(b, slot):
    return [b.get_field(slot, f) for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI)]


@pytest.mark.parametrize("precision", [co.FP32, co.FP64])
def test_graph_gives_back_what_retired_instances_needed(precision):
    """Once instances have retired, their time axis' launches, tiles and shared memory leave the
    graph again within a bounded number of round trips; the instance that stays is the same
    bit for bit as alone."""
    def launches(b):
        n = b.stats()["launches"]
        b.run_round_trips(1)
        return b.stats()["launches"] - n

    cfg = config(16, 16, 32, precision, total_rt=99)
    alone = co.Batch(precision, 1, 8 << 30, tuning=TUNING)
    s = alone.add(cfg)
    alone.init_fields(s, cfg, 3, 0.02, idler_copy=True)
    want = launches(alone)
    b = co.Batch(precision, 4, 8 << 30, tuning=TUNING)
    stay = b.add(cfg)
    b.init_fields(stay, cfg, 3, 0.02, idler_copy=True)
    for nx, nt in ((128, 72), (20, 48), (16, 24)):  # other time axes, a generic axis, many tiles
        c = config(nx, 32, nt, precision, total_rt=99, flags=co.DISPERSION)
        slot = b.add(c)
        b.init_fields(slot, c, 4, 0.02)
        b.run_round_trips(1)
        b.remove(slot)
    assert launches(b) > want
    while launches(b) > want and b.info(stay)["round_trips"] < 90:
        pass
    assert launches(b) == want
    alone.run_round_trips(b.info(stay)["round_trips"] - 1)
    for x, y in zip(fields(b, stay), fields(alone, s)):
        assert np.array_equal(x, y)
    alone.close()
    b.close()


def test_instance_that_cannot_run_leaves_no_trace():
    """An instance whose tile fits shared memory only without the batch's descriptor beside it
    fails the round trip; without it the batch goes on."""
    b = co.Batch(co.FP64, 2, 8 << 30, tuning=dict(TUNING, t=dict(threads=128, tile=4840, r1=4)))
    cfg = config(16, 16, 32)
    s = b.add(cfg)
    b.init_fields(s, cfg, 5, 0.02, idler_copy=True)
    b.run_round_trips(1)
    wide = config(605, 4, 8, flags=co.DISPERSION)  # a 605 x 8 tile of three fields: 232320 bytes
    bad = b.add(wide)
    b.init_fields(bad, wide, 5, 0.02)
    with pytest.raises(co.OpoError) as e:
        b.run_round_trips(1)
    assert e.value.code == co.OPO_ERR_INVALID
    b.remove(bad)
    b.run_round_trips(1)
    for x, y in zip(fields(b, s), standalone(cfg, 2, 5)):
        assert np.array_equal(x, y)
    b.close()

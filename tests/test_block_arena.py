"""A batch's block arena (cuopo3d_b200/csrc/block_arena.h): host code, checked on the CPU with counted
allocations (budget, idle bound, contents of moved blocks, failing allocations); and on the
GPU through the batch: instances whose blocks moved equal standalone solvers bit for bit, and
the device memory that the batch takes stays within its budget."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import cuopo3d_b200 as co

HERE = os.path.dirname(os.path.abspath(__file__))
TUNING = {k: dict(threads=128, tile=1024, r1=4) for k in "txy"}


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_arena_on_the_host(tmp_path):
    exe = str(tmp_path / "arena")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", os.path.join(HERE, "native", "arena_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def config(nx, ny, nt, **over):
    kw = dict(nx=nx, ny=ny, nt=nt, nz=4, LX=300.0, LY=300.0, Lcr=3000.0, P=300.0, w0=40.0, FWHM=3.0, t_window=25.0,
              pump_mode="focused-pulsed", total_rt=9, precision=co.FP64,
              flags=co.DISPERSION | co.DIFFRACTION | co.PHYSICS, Lambda=6.5)
    kw.update(over)
    return co.make_config(**kw)


@pytest.mark.gpu
def test_survivors_of_a_slab_move_within_the_budget():
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    small, large = config(32, 32, 96), config(128, 128, 128)  # 6 and 128 MiB of fields, 1 MiB of tables each
    mib = 1 << 20
    budget = (8 * 7 + 90) * mib  # a slab of eight and no room for the large one's 129 beside it
    for cfg in (small, large):  # lazily loaded modules are not the batch's memory
        b = co.Batch(co.FP64, 1, 8 << 30, tuning=TUNING)
        b.init_fields(b.add(cfg), cfg, 1, 0.02, idler_copy=True)
        b.run_round_trips(1)
        b.close()
    before = free()
    b = co.Batch(co.FP64, 9, budget, tuning=TUNING)
    slots = [b.add(small) for _ in range(8)]
    for k, s in enumerate(slots):
        b.init_fields(s, small, 40 + k, 0.02, idler_copy=True)
    b.run_round_trips(1)
    for k in (0, 1, 2, 4, 5, 6):
        b.remove(slots[k])
    s = b.add(large)  # 14 + 129 MiB charged
    b.init_fields(s, large, 60, 0.02, idler_copy=True)
    assert b.stats()["used"] <= budget
    assert before - free() <= budget + 8 * mib
    b.run_round_trips(1)
    for slot, cfg, seed, nrt in ((slots[3], small, 43, 2), (slots[7], small, 47, 2), (s, large, 60, 1)):
        params, _ = co.derive(cfg)
        _, w = co.time_freq(cfg.nt, params.t_window)
        sim = co.Simulation(params, w)
        sim.set_tuning(TUNING)
        sim.set_plane_pass(0)
        sim.init_fields(cfg, seed, 0.02, idler_copy=True)
        sim.run_round_trips(nrt)
        for f in (co.FIELD_AP, co.FIELD_AS, co.FIELD_AI):
            assert np.array_equal(b.get_field(slot, f), sim.get_field(f))
        sim.close()
    b.close()

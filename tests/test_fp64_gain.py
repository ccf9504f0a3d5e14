"""Gain of the FP64 transform pairs (cuopo3d_b200/csrc/fft_gain.h): the compensation's network against
dense operators with the kernels' constants (host), and a crystal without loss or pump on
the GPU, whose white signal must keep its power.  Bound per step: a table entry's components are
rounded by at most 2^-53 of themselves, its squared modulus by 1.28e-16 r.m.s. at most, the
mean over an axis' n entries by that / sqrt(n); five times the three axes' together.  (The
uncompensated pairs of 64 points gain 1.3e-16 each, those of 36 lose 1.9e-16.)"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import cuopo3d_b200 as co

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="nvcc not available")
def test_fp64_pair_gain_compensation(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "gain64")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets",
                    os.path.join(HERE, "native", "gain64_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("n", [36, 64])
def test_power_without_loss(n):
    steps = 400
    cfg = co.make_config(nx=n, ny=n, nt=n, nz=steps + 1, n_steps=steps, LX=800.0, LY=800.0, Lcr=20000.0, P=1.0, w0=60.0,
                         FWHM=2.0, t_window=40.0, pump_mode="focused-pulsed", alpha=(0.0, 0.0, 0.0), precision=co.FP64)
    params, _ = co.derive(cfg)
    _, w = co.time_freq(n, params.t_window)
    sim = co.Simulation(params, w)
    zero = np.zeros((n, n, n), dtype=np.complex128)
    s0 = co.noise(17, 1.0, zero.size).reshape(zero.shape)
    for which, arr in ((co.FIELD_API, zero), (co.FIELD_AP, zero), (co.FIELD_AS, s0), (co.FIELD_AI, zero)):
        sim.set_field(which, arr)
    sim.run_single_pass()
    power = [np.sum(np.square(a.view(np.float64)), dtype=np.longdouble) for a in (s0, sim.get_field(co.FIELD_AS))]
    drift = float(power[1] / power[0] - 1) / steps
    assert abs(drift) < 5 * 1.28e-16 * np.sqrt(3 / n), drift
    sim.close()

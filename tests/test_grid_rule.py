"""Which uniform grids the FP64 form takes as n dfq (csrc/phenom_acc.h), compiled
for the host: those whose frequencies are that to their own rounding, and no
others.  Runs without a GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("native") / "libgrid_check.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", "-o", lib,
                           os.path.join(ROOT, "tests", "native", "grid_check.cpp")])
    L = ctypes.CDLL(lib)
    L.gwr_dev_error.restype = ctypes.c_double
    return L


def _on_line(rule, f, n0):
    f = np.ascontiguousarray(f)
    return rule.gwr_on_line(f.ctypes.data_as(ctypes.c_void_p), n0, f.size)


@pytest.mark.parametrize("T", [1, 3, 4, 5, 7, 8, 12, 16, 25, 32, 49, 50, 64, 100, 128, 365, 1000, 4096])
@pytest.mark.parametrize("N", [2, 3, 129, 32128])
def test_rounded_grids_are_on_the_line(rule, T, N):
    n0 = 20 * T
    k = np.arange(N)
    for f in (20.0 + k * (1.0 / T), 20.0 + k / T, (n0 + k) / T, (n0 + k) * (1.0 / T), (20.0 + k / T) * (1 + 3e-10)):  # the last: n times another spacing
        assert _on_line(rule, f, n0) == 1


@pytest.mark.parametrize("T", [4, 25, 32, 64])
@pytest.mark.parametrize("off", [1e-12, 1e-10, 1e-9, 1e-8, 2.5e-8])
def test_other_grids_are_not(rule, T, off):
    N, n0 = 32128, 20 * T
    k = np.arange(N)
    f = 20.0 + k * (1.0 / T)
    wave = off * np.sin(k / 500.0)
    for g in (f + off, 20.0 + k / T * (1 + off), f + wave):
        assert _on_line(rule, g, n0) == 0


def test_rounding_times_tc(rule):
    """FP32 products: 2^-23 of the turns, and the 2^-55 turn of the fixed point; up to t_c in GPS seconds."""
    for tc in (1.0, 32.0, 4096.0, 1e6, 1.2e9):
        for dev in np.float32([0.0, 1e-16, 3.3e-15, -1.1e-13, 4.5e-13, -9e-12]):
            err = rule.gwr_dev_error(ctypes.c_double(tc), ctypes.c_float(dev))
            assert err <= abs(tc * float(dev)) * 2.0 ** -22 + 2.0 ** -55, (tc, dev, err)

"""IMRPhenomPv2's J frame where the in-plane spin is nothing or nearly so (csrc/phenom_fast.h), compiled for the
host, against the oracle: J along and against the orbital axis.  Runs without a GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gw_analysis_tools_gb300 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def acc(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("native") / "libacc_check.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", "-o", lib,
                           os.path.join(ROOT, "tests", "native", "acc_check.cpp")])
    L = ctypes.CDLL(lib)
    L.gwa_loglik.restype = ctypes.c_double
    return L


@pytest.mark.parametrize("spin", [0.9, -0.9])  # a heavy mass ratio: J along, J against the axis
@pytest.mark.parametrize("plane", [0.0, 1e-16, 1e-12, 1e-9, 1e-8, 3e-8, 1e-7, 1e-6, 1e-5, 1e-4, 1e-2])
def test_against_oracle(acc, oracle, spin, plane):
    T, n0, N = 8, 160, 1500
    f = 20.0 + np.arange(N) / T
    dets = list(W.DETECTORS3)
    src = W.config1_source()
    data, psd = [W.noise(f, 5 + i) for i in range(3)], [W.analytic_psd(f)] * 3
    idx = (ctypes.c_int * 3)(*[oracle.detector_index(d) for d in dets])
    rng = np.random.default_rng(7)
    for k in range(12):
        az = rng.uniform(0, 2 * np.pi)
        d = dict(src, mass1=rng.uniform(40, 90), mass2=rng.uniform(1, 4), incl_angle=[0.0, np.pi / 2, 0.7, 2.6][k % 4],
                 phiRef=rng.uniform(0, 6), f_ref=[20.0, 100.0][k % 2],
                 spin1=(plane * np.cos(az), plane * np.sin(az), spin), spin2=(0, 0, rng.uniform(-0.9, 0.9)))
        p = oracle.params_from_dict(d)
        ref = oracle.loglik(p, f, dets, data, psd, approximant=1, T_segment=T)
        flag = ctypes.c_int()
        got = acc.gwa_loglik(ctypes.byref(p), 1, ctypes.c_double(T), n0, oracle._dp(f), N, 3, idx, oracle._ptr_array(data),
                             oracle._ptr_array(psd), 2, ctypes.byref(flag))
        assert abs(got - ref) <= 1e-9 * max(1.0, abs(ref)), (d, got, ref)

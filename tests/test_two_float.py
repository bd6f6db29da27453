"""The two-float arithmetic (csrc/two_float.h) and the FP64 form's bins built
on it (csrc/phenom_acc.h), compiled for the host, against long double and the
oracle.  Runs without a GPU."""
import ctypes
import os
import platform
import subprocess

import numpy as np
import pytest

from gw_analysis_tools_gb300 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def acc():
    src = os.path.join(ROOT, "tests", "native", "acc_check.cpp")
    lib = os.path.join(ROOT, "tests", "native", "libgwgpu_acccheck.so")
    csrc = os.path.join(ROOT, "gw_analysis_tools_gb300", "csrc")
    newest = max([os.path.getmtime(src)] + [os.path.getmtime(os.path.join(csrc, f)) for f in os.listdir(csrc)
                                            if f.endswith(".h")])
    if not os.path.exists(lib) or os.path.getmtime(lib) < newest:
        subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", "-o", lib, src])
    L = ctypes.CDLL(lib)
    L.gwa_loglik.restype = ctypes.c_double
    return L


def test_elementary(acc):
    """48-bit pairs: a table entry is rounded to 2^-49, a product or sum to a few 2^-48 = 3.6e-15, and
    each function chains fewer than sixteen of them (the exponent carries z's own rounding, |z| < 8)."""
    out = (ctypes.c_double * 6)()
    acc.gwa_worst(ctypes.c_ulonglong(88172645463325252), 300000, out)
    assert max(out) <= 16 * 2.0 ** -48, list(out)


def _loglik(acc, oracle, p, ap, T, n0, f, N, dets, data, psd, mode=0):
    idx = (ctypes.c_int * len(dets))(*[oracle.detector_index(d) for d in dets])
    flag = ctypes.c_int()
    v = acc.gwa_loglik(ctypes.byref(p), ap, ctypes.c_double(T), n0, oracle._dp(f), N, len(dets), idx,
                       oracle._ptr_array(data), oracle._ptr_array(psd), mode, ctypes.byref(flag))
    return v, flag.value


@pytest.mark.parametrize("T,fmax,ndet", [(4, 300, 1), (8, 1024, 2), (32, 512, 3), (12, 400, 3)])
@pytest.mark.parametrize("ap", [0, 1])
def test_loglik_against_oracle(acc, oracle, T, fmax, ndet, ap):
    """The FP64 bound of the likelihood entry points, 1e-9 relative, over prior draws, an aligned
    source without any in-plane spin, and a mass ratio that sends the phase back to FP64."""
    n0, df, N = 20 * T, 1.0 / T, T * (fmax - 20)
    f = 20.0 + np.arange(N) * df  # T = 12: not n df to the last bit
    dets = list(W.DETECTORS3)[:ndet]
    src = W.config1_source()
    injp = oracle.params_from_dict(dict(src, tc=T - src["tc"]))
    data = [oracle.detector_response(f, injp, d) + W.noise(f, 5 + i) for i, d in enumerate(dets)]
    psd = [W.analytic_psd(f)] * ndet
    draws = W.prior_draws(10, 3 + T, precessing=bool(ap)) + [src, dict(src, spin1=(0, 0, 0), spin2=(0, 0, 0)),
                                                              dict(src, mass1=70.0, mass2=1.2)]
    flags = []
    for d in draws:
        p = oracle.params_from_dict(d)
        ref = oracle.loglik(p, f, dets, data, psd, approximant=ap, T_segment=T)
        got, flag = _loglik(acc, oracle, p, ap, T, n0, f, N, dets, data, psd)
        assert abs(got - ref) <= 1e-9 * max(1.0, abs(ref)), (d, got, ref)
        other, _ = _loglik(acc, oracle, p, ap, T, n0, f, N, dets, data, psd, mode=1)
        assert abs(other - ref) <= 1e-9 * max(1.0, abs(ref)), (d, other, ref)
        flags.append(flag)
    assert min(flags) == 0 and flags[-1] == 1


@pytest.mark.parametrize("ap", [0, 1])
def test_fast_prologue(acc, oracle, ap):
    """phenom_fast.h's prologue at its branches: equal and swapped masses, f_ref past the inspiral, no time or
    phase shift, the sky average, the other ringdown fit, aligned and reduced Pv2 spins, a face-on source."""
    T, n0, N = 8, 160, 4000
    f = 20.0 + np.arange(N) / T
    dets = list(W.DETECTORS3)
    src = W.config1_source()
    inj = oracle.params_from_dict(dict(src, tc=T - src["tc"]))
    data = [oracle.detector_response(f, inj, d) + W.noise(f, 15 + i) for i, d in enumerate(dets)]
    psd = [W.analytic_psd(f)] * 3
    kinds = [dict(), dict(mass2=36.0), dict(mass1=29.0, mass2=36.0), dict(f_ref=300.0), dict(mass1=150.0, mass2=90.0, f_ref=60.0),
             dict(shift_time=0), dict(shift_phase=0), dict(sky_average=1), dict(dep_postmerger=1), dict(incl_angle=0.0),
             dict(spin1=(0, 0, 0.0), spin2=(0, 0, 0.0)), dict(chip=0.4, phip=1.0), dict(mass1=80.0, mass2=5.0)]
    for k in kinds:
        for base in (src, W.prior_draws(1, 77, precessing=bool(ap))[0]):
            d = dict(base, **k)
            p = oracle.params_from_dict({a: b for a, b in d.items() if a not in ("shift_time", "shift_phase", "sky_average",
                                                                                 "dep_postmerger", "chip", "phip")})
            for a in ("shift_time", "shift_phase", "sky_average", "dep_postmerger", "chip", "phip"):
                if a in d:
                    setattr(p, a, d[a])
            ref = oracle.loglik(p, f, dets, data, psd, approximant=ap, T_segment=T)
            got, _ = _loglik(acc, oracle, p, ap, T, n0, f, N, dets, data, psd, mode=2)
            assert (np.isnan(ref) and np.isnan(got)) or abs(got - ref) <= 1e-9 * max(1.0, abs(ref)), (k, got, ref)

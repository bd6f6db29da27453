"""IMRPhenomPv2 with no in-plane spin, or nearly none, J along and against the orbital axis: the FP64 calls
against the oracle."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston", "Virgo")


@pytest.mark.parametrize("plane", [0.0, 1e-16, 1e-12, 1e-10, 1e-5, 1e-2])
def test_log_likelihoods(gpu_ctx, oracle, plane):
    T, N = 8.0, 1500
    f = 20.0 + np.arange(N) / T
    psd, data = [W.analytic_psd(f)] * 3, [W.noise(f, 5 + i) for i in range(3)]
    hs = [gpu_ctx.register_data(d, f, data[i], psd[i]) for i, d in enumerate(DETS)]
    rng, draws = np.random.default_rng(7), []
    for k in range(24):
        az = rng.uniform(0, 2 * np.pi)
        draws.append(dict(W.config1_source(), mass1=rng.uniform(40, 90), mass2=rng.uniform(1, 4), phiRef=rng.uniform(0, 6),
                          incl_angle=[0.0, np.pi / 2, 0.7, 2.6][k % 4], f_ref=[20.0, 100.0][k % 2],
                          spin1=(plane * np.cos(az), plane * np.sin(az), 0.9 if k % 3 else -0.9),
                          spin2=(0, 0, rng.uniform(-0.9, 0.9))))
    ref = np.array([oracle.loglik(oracle.params_from_dict(d), f, list(DETS), data, psd, approximant=1, T_segment=T)
                    for d in draws])
    mref = np.array([oracle.maximized_loglik_intrinsic(d, f, data, psd, approximant=1) for d in draws])
    try:
        out, st = gpu_ctx.loglik_batch(G.params_array(draws), 1, hs, T, G.PREC_FP64)
        assert np.all(st == 0) and np.all(np.abs(out - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
        plain = np.array([gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**d), "IMRPhenomPv2", hs, T) for d in draws])
        assert np.all(np.abs(plain - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
        out, st = gpu_ctx.maximized_loglik_batch(G.params_array(draws), hs, 1)
        assert np.all(st == 0) and np.all(np.abs(out - mref) <= 1e-9 * np.maximum(1.0, np.abs(mref)))
    finally:
        for h in hs:
            gpu_ctx.release_data(h)

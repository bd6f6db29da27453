"""FP64 calls on streams whose weights or data span more than FP32's exponents, against the oracle."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston")


def _streams(kind, f):
    psd, data = W.analytic_psd(f), [W.noise(f, 3 + i) for i in range(2)]
    beyond = f > 900.0
    if kind == "filled with 1e-100":
        psd = np.where(beyond, 1e-100, psd)
    elif kind == "filled with 1e-62":
        psd = np.where(beyond, 1e-62, psd)
    elif kind == "filled with one":
        psd = np.where(beyond, 1.0, psd)
    elif kind == "spike":  # one bin of the data
        data = [np.where(np.arange(f.size) == f.size - 3, 1e25, d) for d in data]
    elif kind == "masked below 30 Hz":
        psd = np.where(f < 30.0, 1.0, psd)
    elif kind == "infinite below 30 Hz":
        psd = np.where(f < 30.0, np.inf, psd)
    elif kind == "signal alone":
        data = [np.exp(-((f - 100.0) / 20.0) ** 2) * 1e-22 * np.exp(0.3j * f) for _ in data]
    return psd, data


@pytest.mark.parametrize("kind", ["filled with 1e-100", "filled with 1e-62", "filled with one", "spike", "masked below 30 Hz",
                                  "infinite below 30 Hz", "signal alone"])
@pytest.mark.parametrize("nodes", [False, True])
@pytest.mark.parametrize("ap", [0, 1])
def test_log_likelihoods(gpu_ctx, oracle, kind, nodes, ap):
    T, N = 8.0, 8000
    f = 20.0 + np.arange(N) / T
    f = f + 0.37 / T if nodes else f
    psd, data = _streams(kind, f)
    hs = [gpu_ctx.register_data(d, f, data[i], psd) for i, d in enumerate(DETS)]
    # heavy enough for every cut to lie below the filled bins
    draws = [dict(d, mass1=50.0 + i, mass2=30.0) for i, d in enumerate(W.prior_draws(4, 9, precessing=bool(ap)))]
    ref = np.array([oracle.loglik(oracle.params_from_dict(d), f, list(DETS), data, [psd] * 2, approximant=ap, T_segment=T)
                    for d in draws])
    mref = np.array([oracle.maximized_loglik_intrinsic(d, f, data, [psd] * 2, approximant=ap) for d in draws])
    try:
        out, st = gpu_ctx.loglik_batch(G.params_array(draws), ap, hs, T, G.PREC_FP64)
        assert np.all(st == 0) and np.all(np.abs(out - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
        for d, r in zip(draws, ref):
            got = gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**d), "IMRPhenomPv2" if ap else "IMRPhenomD", hs, T)
            assert abs(got - r) <= 1e-9 * max(1.0, abs(r))
        out, st = gpu_ctx.maximized_loglik_batch(G.params_array(draws), hs, ap)
        assert np.all(st == 0) and np.all(np.abs(out - mref) <= 1e-9 * np.maximum(1.0, np.abs(mref)))
    finally:
        for h in hs:
            gpu_ctx.release_data(h)


def test_fisher_moments(gpu_ctx):
    """Weights filled in beyond the cut change no element: the sums end there."""
    T, N = 8.0, 8000
    f = 20.0 + np.arange(N) / T
    draws = [dict(d, mass1=50.0 + i, mass2=30.0) for i, d in enumerate(W.prior_draws(4, 9))]
    kw = dict(order=2, epsilon=1e-6, step_mode=1, precision=G.PREC_FP64, algorithm=G.FISHER_MOMENTS, covariance=False)
    got = []
    for kind in ("as it is", "filled with 1e-100"):
        hs = [gpu_ctx.register_data(d, f, np.zeros(N, complex), _streams(kind, f)[0]) for d in DETS]
        F, _, st = gpu_ctx.fisher_batch_ex(G.params_array(draws), 1, hs, **kw)
        for h in hs:
            gpu_ctx.release_data(h)
        assert np.all(st == 0)
        got.append(F)
    for a, b in zip(*got):
        s = np.sqrt(np.diag(a))
        assert np.max(np.abs(a - b) / np.outer(s, s)) <= 1e-11

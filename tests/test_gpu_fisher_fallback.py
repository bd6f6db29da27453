"""Fisher calls whose sources two floats cannot all hold: the whole chunk takes the FP64 sums."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [500, 4097, 9000])
@pytest.mark.parametrize("order,eps,mode", [(2, 1e-6, 1), (4, 1e-8, 0)])
def test_same_sums_as_the_call_with_an_inverse(gpu_ctx, N, order, eps, mode):
    """A ringdown beyond 2^24 bins beside ordinary sources: to the bit the matrices of the call that
    always takes FP64 sums."""
    T = 8
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    hs = [gpu_ctx.register_data(d, f, np.zeros(N, complex), psd) for d in ("Hanford", "Livingston", "Virgo")]
    draws = [dict(d, mass1=36.0 + i, mass2=20.0 + i) for i, d in enumerate(W.prior_draws(6, 17))]
    beyond = dict(draws[0], mass1=2e-6, mass2=1e-6)
    kw = dict(order=order, epsilon=eps, step_mode=mode, precision=G.PREC_FP64, algorithm=G.FISHER_MOMENTS)
    try:
        got, _, st = gpu_ctx.fisher_batch_ex(G.params_array(draws + [beyond]), 1, hs, covariance=False, **kw)
        ref, _, sr = gpu_ctx.fisher_batch_ex(G.params_array(draws + [beyond]), 1, hs, covariance=True, **kw)
        same = sr[:-1] == 0  # a matrix without an inverse is made again by the reference algorithm
        assert np.all(st[:-1] == 0) and np.sum(same) >= 3
        assert np.array_equal(got[:-1][same], ref[:-1][same])
    finally:
        for h in hs:
            gpu_ctx.release_data(h)

"""The transform tables that a context keeps for one grid length, when a call at
another length does not get its memory."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
N1, M1, N2, M2 = 4099, 8192, 70001, 262144  # grid lengths with a large prime factor and their padded lengths


def _stream(ctx, N, T):
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    psd[-1] *= 1e80  # a weight out of the other bins' range: the stream keeps FP64 bins
    return ctx.register_data("Hanford", f, W.noise(f, 3), psd)


def _calls(budget):
    """Log L at N1, what a call at N2 raises, log L at N1 again; the bytes held after the first."""
    ctx = G.Context(0, hbm_budget=budget)
    try:
        short, long = _stream(ctx, N1, 8), _stream(ctx, N2, 64)
        p = G.params_array(W.prior_draws(3, 5))
        first = ctx.maximized_loglik_batch(p, [short], 0)[0]
        held, failed = ctx.bytes_in_use(), None
        try:
            ctx.maximized_loglik_batch(p, [long], 0)
        except Exception as e:
            failed = str(e)
        again = ctx.maximized_loglik_batch(p, [short], 0)[0]
        return first, failed, again, held
    finally:
        ctx.close()


@pytest.mark.parametrize("part", [0.25, 0.5, 0.75])
def test_failed_longer_call(part):
    """The longer chirp fits the budget, its FP32 copy does not: the shorter length's tables are made again."""
    first, failed, _, held = _calls(0)
    assert failed is None
    budget = held + 16 * (M2 - M1) + int(part * 8 * (M2 + N2 - M1 - N1))
    got, failed, again, _ = _calls(budget)
    assert failed is not None and "budget" in failed.lower()
    assert np.array_equal(got, first) and np.array_equal(again, first)

"""The maximised likelihood's search when it gives up: one more pass at most."""
import time

import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ap", [0, 1])
def test_a_flat_spectrum_costs_one_search(oracle, monkeypatch, ap):
    """Data at a single bin: every lag scores the same, the search keeps none.  Its own pass (products,
    transforms and candidates in FP32) is a part of the FP64 transforms' time, so that with it the call
    stays below twice that; and the results are theirs."""
    T, N = 8, 8000
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    data = np.zeros(N, complex)
    data[1000] = 1e-22
    draws = W.prior_draws(64, 5, precessing=bool(ap))
    best, outs = [], []
    for mode in ("search", "fp64"):
        monkeypatch.setenv("GWGPU_MAXLL", mode)
        ctx = G.Context(0)
        try:
            hs = [ctx.register_data(d, f, data, psd) for d in ("Hanford", "Livingston", "Virgo")]
            p, times = G.params_array(draws), []
            for _ in range(12):
                t = time.perf_counter()
                out, st = ctx.maximized_loglik_batch(p, hs, ap)
                times.append(time.perf_counter() - t)
            assert np.all(st == 0)
            best.append(min(times))
            outs.append(out)
        finally:
            ctx.close()
    assert np.all(np.abs(outs[0] - outs[1]) <= 1e-10 * np.maximum(1e-12, np.abs(outs[1])))
    ref = [oracle.maximized_loglik_intrinsic(d, f, [data] * 3, [psd] * 3, approximant=ap) for d in draws[:4]]
    assert np.all(np.abs(outs[0][:4] - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
    assert best[0] < 2.0 * best[1], best

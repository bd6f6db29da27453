"""Device memory that a context keeps for the FP64 form's two-float bins."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_tables_of_slowly_growing_grids(oracle):
    """Grids each a little longer than any before, registered and released: what stays allocated is
    bounded by a few times the longest one's tables, and log L on the last grid is right."""
    ctx = G.Context(0)
    try:
        T, held = 64.0, []
        for N in range(70000, 74000, 200):
            f = 20.0 + np.arange(N) / T
            psd, data = W.analytic_psd(f), W.noise(f, 3)
            h = ctx.register_data("Hanford", f, data, psd)
            if N == 73800:
                draws = W.prior_draws(3, 4)
                ref = [oracle.loglik(oracle.params_from_dict(d), f, ["Hanford"], [data], [psd], T_segment=T) for d in draws]
                out, st = ctx.loglik_batch(G.params_array(draws), 0, [h], T, G.PREC_FP64)
                assert np.all(st == 0) and np.all(np.abs(out - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
            ctx.release_data(h)
            held.append(ctx.bytes_in_use())
        assert held[-1] <= 4 * held[0]
    finally:
        ctx.close()


@pytest.mark.parametrize("prec", [G.PREC_MIXED, G.PREC_FP64])
def test_registration_that_fails(prec):
    """A longer grid that gets its tables and not its own arrays, or neither: calls on the streams that
    were there (replayed launches among them) go on as before."""
    T, N, N2 = 8.0, 3000, 150000
    f, g = 20.0 + np.arange(N) / T, 20.0 + np.arange(N2) / 64.0
    psd, data = W.analytic_psd(f), W.noise(f, 3)
    gpsd, gdata = W.analytic_psd(g), W.noise(g, 4)
    p = G.params_array(W.prior_draws(6, 4))

    def run(budget):
        ctx = G.Context(0, hbm_budget=budget)
        try:
            h = ctx.register_data("Hanford", f, data, psd)
            call = lambda: ctx.loglik_batch(p, 0, [h], T, prec)
            out = [call()[0] for _ in range(3)]
            held, failed = ctx.bytes_in_use(), 0
            try:
                ctx.register_data("Hanford", g, gdata, gpsd)
            except Exception:
                failed = 1
            after = ctx.bytes_in_use()
            for _ in range(2):
                v, st = call()
                assert np.all(st == 0)
                out.append(v)
            if failed or not budget:
                assert all(np.array_equal(v, out[0]) for v in out)
            else:  # the longer grid may have taken the place of the two-float arrays
                assert all(np.all(np.abs(v - out[0]) <= 1e-9 * np.maximum(1.0, np.abs(out[0]))) for v in out)
            return held, after - held, failed
        finally:
            ctx.close()

    held, need, failed = run(0)
    assert not failed
    parts = [run(held + int(need * x))[2] for x in np.linspace(0.0, 1.0, 9)]
    assert parts[0] == 1 and parts[-1] == 0

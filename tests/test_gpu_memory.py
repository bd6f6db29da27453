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

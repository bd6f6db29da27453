"""A request whose model ends below the grid: log L is zero, whatever its phase would have been."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ap", [0, 1])
@pytest.mark.parametrize("off", [0.0, 1e-8, 0.03])
def test_zero(gpu_ctx, oracle, ap, off):
    T, N = 8.0, 700
    f = 100.0 + off + np.arange(N) / T
    psd, data = W.analytic_psd(f), W.noise(f, 3)
    h = gpu_ctx.register_data("Hanford", f, data, psd)
    src = W.config1_source()
    beyond = dict(src, mass1=2000.0, mass2=500.0)
    draws = [beyond] + [dict(beyond, **{k: v}) for k, v in (("f_ref", 0.0), ("f_ref", -20.0), ("tc", np.nan))]
    draws += [dict(src, tc=np.nan), src]
    if ap:  # f_ref <= 0 is outside the domain of IMRPhenomPv2
        draws = [draws[0], draws[3], draws[4], draws[5]]
    try:
        out, st = gpu_ctx.loglik_batch(G.params_array(draws), ap, [h], T, G.PREC_FP64)
        ref = oracle.loglik(oracle.params_from_dict(src), f, ["Hanford"], [data], [psd], approximant=ap, T_segment=T)
        assert np.all(st == 0) and np.all(out[:-2] == 0.0) and np.isnan(out[-2])
        assert abs(out[-1] - ref) <= 1e-9 * max(1.0, abs(ref))
        plain = [gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**d), "IMRPhenomPv2" if ap else "IMRPhenomD", [h], T)
                 for d in draws]
        assert np.all(np.array(plain[:-2]) == 0.0) and np.isnan(plain[-2])
    finally:
        gpu_ctx.release_data(h)

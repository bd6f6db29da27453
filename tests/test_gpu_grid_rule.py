"""FP64 likelihoods on uniform grids that are not whole multiples of their
spacing: offsets and drifts that registration still calls uniform, on every
route that takes two-float bins, against the oracle."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston", "Virgo")
RTOL = 1e-9  # the FP64 bound of the likelihood entry points


def _grid(kind, T, N):
    k = np.arange(N)
    f = 20.0 + k / T
    if isinstance(kind, float):
        return f + kind  # 1e-9 .. 8e-7 of a bin
    if kind == "stretched":
        return 20.0 + k / T * (1 + 7e-10)
    return f + 4e-10 / T * (1 + k) * np.sin(k / 300.0)  # "drifting"


@pytest.mark.parametrize("kind", [1e-10, 1e-9, 1e-8, 2.5e-8, "stretched", "drifting"])
@pytest.mark.parametrize("ap", [0, 1])
def test_grids_off_the_line(gpu_ctx, oracle, kind, ap):
    T, N = 32.0, 8128
    f = _grid(kind, T, N)
    src = W.config1_source()
    inj = oracle.params_from_dict(dict(src, tc=T - src["tc"]))
    psd = [W.analytic_psd(f)] * 3
    data = [oracle.detector_response(f, inj, d) + W.noise(f, 5 + i) for i, d in enumerate(DETS)]
    hs = [gpu_ctx.register_data(d, f, data[i], psd[i]) for i, d in enumerate(DETS)]
    # a light binary (the largest phases), one whose phase falls back to FP64, one with its cut inside the grid
    draws = [src, dict(src, mass1=1.6, mass2=1.2), dict(src, mass1=70.0, mass2=1.2), dict(src, mass1=150.0, mass2=90.0)]
    draws += W.prior_draws(4, 31, precessing=bool(ap))
    par = G.params_array(draws)
    ref = np.array([oracle.loglik(oracle.params_from_dict(d), f, list(DETS), data, psd, approximant=ap, T_segment=T)
                    for d in draws])
    mref = np.array([oracle.maximized_loglik_intrinsic(d, f, data, psd, approximant=ap) for d in draws])
    bound = lambda r: RTOL * np.maximum(1.0, np.abs(r))
    try:
        out, st = gpu_ctx.loglik_batch(par, ap, hs, T, G.PREC_FP64)
        assert np.all(st == 0) and np.all(np.abs(out - ref) <= bound(ref)), np.abs(out / ref - 1).max()
        plain = np.array([gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**d), "IMRPhenomPv2" if ap else "IMRPhenomD", hs, T)
                          for d in draws])
        assert np.all(np.abs(plain - ref) <= bound(ref)), np.abs(plain / ref - 1).max()
        out, st = gpu_ctx.maximized_loglik_batch(par, hs, ap)
        assert np.all(st == 0) and np.all(np.abs(out - mref) <= bound(mref)), np.abs(out / mref - 1).max()
        # beside a grid on the line, in one call
        g = 20.0 + np.arange(N) / T
        gd = [W.noise(g, 50 + i) for i in range(3)]
        gh = [gpu_ctx.register_data(d, g, gd[i], W.analytic_psd(g)) for i, d in enumerate(DETS)]
        alone, _ = gpu_ctx.loglik_batch(par, ap, gh, T, G.PREC_FP64)
        both, st = gpu_ctx.loglik_batch(G.params_array(draws + draws), ap, np.array([hs] * len(draws) + [gh] * len(draws)),
                                        T, G.PREC_FP64)
        for h in gh:
            gpu_ctx.release_data(h)
        assert np.all(st == 0) and np.all(np.abs(both - np.concatenate([ref, alone])) <= bound(np.concatenate([ref, alone])))
    finally:
        for h in hs:
            gpu_ctx.release_data(h)

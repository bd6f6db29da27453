"""The FP64 form's FP64 bins (streams without two-float arrays): IMRPhenomD from its coefficients on the grid and
the arrival times' rotations as products, at the edges of passes, tiles and blocks, against the oracle."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston", "Virgo", "Kagra")
RTOL = 1e-9  # the FP64 bound of the likelihood entry points


@pytest.fixture(scope="module")
def ctx():
    """A context whose budget leaves no room for the two-float tables (80 bytes for each of 65,537 bins)."""
    probe = G.Context(0)
    f = 20.0 + np.arange(64) / 4.0
    probe.register_data("Hanford", f, np.zeros(64, complex), W.analytic_psd(f))
    used = probe.bytes_in_use()
    probe.close()
    c = G.Context(0, hbm_budget=used - (1 << 18))
    yield c
    c.close()


@pytest.mark.parametrize("T,N,ndet", [(8, 2, 1), (8, 127, 3), (8, 129, 4), (4, 255, 2), (4, 257, 1), (25, 2049, 3),
                                      (16, 4097, 2)])
def test_batch_and_plain(ctx, oracle, T, N, ndet):
    f = 20.0 + np.arange(N) * (1.0 / T)
    src = W.config1_source()
    psd = [W.analytic_psd(f) * (1 + 0.2 * i) for i in range(ndet)]
    inj = oracle.params_from_dict(dict(src, tc=T - src["tc"]))
    data = [oracle.detector_response(f, inj, d) + W.noise(f, 7 + i) for i, d in enumerate(DETS[:ndet])]
    hs = [ctx.register_data(d, f, data[i], psd[i]) for i, d in enumerate(DETS[:ndet])]
    # f_ref past the inspiral, a cut inside the grid, a light binary, and precessing ones beside them
    draws = [src, dict(src, f_ref=300.0), dict(src, mass1=150.0, mass2=90.0), dict(src, mass1=1.6, mass2=1.2)]
    draws += W.prior_draws(3, N) + W.prior_draws(3, N + 1, precessing=True)
    aps = [0] * 7 + [1] * 3
    ref = np.array([oracle.loglik(oracle.params_from_dict(x), f, list(DETS[:ndet]), data, psd, approximant=a,
                                  T_segment=float(T)) for x, a in zip(draws, aps)])
    bound = RTOL * np.maximum(1.0, np.abs(ref))
    try:
        for tile in (0, 256, 768):
            ctx.set_tile(tile)
            out, st = ctx.loglik_batch(G.params_array(draws), aps, hs, float(T), G.PREC_FP64)
            assert np.all(st == 0) and np.all(np.abs(out - ref) <= bound), (tile, np.abs(out - ref).max())
        for x, a, r, b in zip(draws, aps, ref, bound):
            got = ctx.mcmc_likelihood_extrinsic(G.gen_params(**x), "IMRPhenomPv2" if a else "IMRPhenomD", hs, float(T))
            assert abs(got - r) <= b
    finally:
        ctx.set_tile(0)
        for h in hs:
            ctx.release_data(h)


def test_beside_a_stream_that_is_not_finite(gpu_ctx, oracle):
    """One datum that is not a number leaves a batch's other requests as they are."""
    T, N = 8.0, 1500
    f = 20.0 + np.arange(N) / T
    psd, data = W.analytic_psd(f), W.noise(f, 3)
    bad = data.copy()
    bad[-1] = np.nan
    good, nan = (gpu_ctx.register_data("Virgo", f, x, psd) for x in (data, bad))
    draws = W.prior_draws(5, 8)
    ref = np.array([oracle.loglik(oracle.params_from_dict(x), f, ["Virgo"], [data], [psd], T_segment=T) for x in draws])
    try:
        out, st = gpu_ctx.loglik_batch(G.params_array(draws + draws), 0, np.array([[good]] * 5 + [[nan]] * 5), T, G.PREC_FP64)
        assert np.all(st == 0) and np.all(np.abs(out[:5] - ref) <= RTOL * np.maximum(1.0, np.abs(ref)))
        assert np.all(np.isnan(out[5:]))
    finally:
        gpu_ctx.release_data(good)
        gpu_ctx.release_data(nan)

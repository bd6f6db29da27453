"""The FP64 form's two-float bins on the device (csrc/acc.cu): batched and plain
log L against the oracle at the sizes where tiles, blocks and grids end, on
grids whose frequencies are rounded, with different weights per detector, and
with requests and streams that take another branch."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston", "Virgo", "Kagra")
RTOL = 1e-9  # the FP64 bound of the likelihood entry points


def _network(ctx, oracle, T, N, ndet, same_psd=True, seed=3):
    f = 20.0 + np.arange(N) * (1.0 / T)
    src = W.config1_source()
    inj = oracle.params_from_dict(dict(src, tc=T - src["tc"]))
    rng = np.random.default_rng(seed)
    psd = [W.analytic_psd(f) * (1.0 if same_psd else 1.0 + 0.3 * i) for i in range(ndet)]
    data = [oracle.detector_response(f, inj, d) + np.sqrt(psd[i] * T / 4) * (rng.standard_normal(N) + 1j * rng.standard_normal(N))
            for i, d in enumerate(DETS[:ndet])]
    return f, data, psd, [ctx.register_data(d, f, data[i], psd[i]) for i, d in enumerate(DETS[:ndet])]


def _close(got, ref):
    return np.all(np.abs(np.asarray(got) - ref) <= RTOL * np.maximum(1.0, np.abs(ref)))


@pytest.mark.parametrize("T,N,ndet,same", [(8, 2, 1, True), (8, 3, 2, True), (8, 127, 3, True), (8, 129, 4, False),
                                           (4, 255, 3, False), (4, 257, 1, True), (16, 4095, 2, False),
                                           (12, 4097, 3, True), (25, 9001, 3, False), (32, 32128, 2, True)])
def test_batch_and_plain(gpu_ctx, oracle, T, N, ndet, same):
    f, data, psd, hs = _network(gpu_ctx, oracle, T, N, ndet, same)
    try:
        # a near-aligned source with no in-plane spin and an extreme mass ratio beside the draws
        src = W.config1_source()
        d = [src, dict(src, mass1=70.0, mass2=1.2)] + W.prior_draws(5, N)
        p = [dict(src, spin1=(0, 0, 0), spin2=(0, 0, 0)), dict(src, mass1=70.0, mass2=1.2, spin1=(0.4, 0.1, 0.2))]
        p += W.prior_draws(5, N + 1, precessing=True)
        draws = [x for pair in zip(d, p) for x in pair]
        aps = [0, 1] * len(d)
        ref = np.array([oracle.loglik(oracle.params_from_dict(x), f, list(DETS[:ndet]), data, psd, approximant=a,
                                      T_segment=float(T)) for x, a in zip(draws, aps)])
        for tile in (0, 256, 512):
            gpu_ctx.set_tile(tile)
            out, st = gpu_ctx.loglik_batch(G.params_array(draws), aps, hs, float(T), G.PREC_FP64)
            assert np.all(st == 0) and _close(out, ref), (tile, np.abs(out - ref).max())
        for x, a, r in zip(draws, aps, ref):
            m = "IMRPhenomPv2" if a else "IMRPhenomD"
            assert _close(gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**x), m, hs, float(T)), r)
    finally:
        gpu_ctx.set_tile(0)
        for h in hs:
            gpu_ctx.release_data(h)


def test_weighted_uniform_grid_and_bad_requests(gpu_ctx, oracle):
    """Integration weights on a uniform grid, and requests outside the model's domain beside good ones."""
    T, N = 8.0, 1500
    f = 20.0 + np.arange(N) / T
    rng = np.random.default_rng(5)
    w = rng.uniform(0.5, 1.5, N) / T
    psd = W.analytic_psd(f)
    data = W.noise(f, 9)
    h = gpu_ctx.register_data("Hanford", f, data, psd, weights=w)
    try:
        draws = W.prior_draws(6, 8)
        ref = np.array([oracle.loglik_gl(oracle.params_from_dict(x), f, ["Hanford"], [data], [psd], [w], T_segment=T)
                        for x in draws])
        bad = [dict(draws[0], mass1=-1.0), dict(draws[1], mass1=float("nan"))]
        out, st = gpu_ctx.loglik_batch(G.params_array(draws + bad), 0, [h], T, G.PREC_FP64)
        assert np.all(st[:6] == 0) and _close(out[:6], ref)
        assert np.all(st[6:] != 0) and np.all(np.isnan(out[6:]))
    finally:
        gpu_ctx.release_data(h)


@pytest.mark.parametrize("ap,key,val,want", [
    (0, "tc", float("nan"), "nan"), (1, "tc", float("nan"), "nan"), (0, "tc", float("inf"), "nan"),
    (0, "phiRef", float("nan"), "nan"), (0, "f_ref", float("nan"), "nan"), (0, "f_ref", 0.0, "nan"),
    (1, "RA", float("nan"), "nan"), (0, "Luminosity_Distance", 1e-300, "-inf"), (1, "Luminosity_Distance", 1e-300, "-inf")])
def test_non_finite_parameters(gpu_ctx, ap, key, val, want):
    """A phase that is not a number reaches log L though angles are integers; an infinite
    amplitude squared outweighs the finite cross term."""
    f = 20.0 + np.arange(4000) / 8.0
    psd = W.analytic_psd(f)
    hs = [gpu_ctx.register_data(d, f, W.noise(f, 9 + i), psd) for i, d in enumerate(DETS[:2])]
    x = dict(W.prior_draws(1, 8, precessing=bool(ap))[0], **{key: val})
    out, st = gpu_ctx.loglik_batch(G.params_array([x]), ap, hs, 8.0, G.PREC_FP64)
    assert np.array_equal(out, [float(want)], equal_nan=True) and st[0] == 0
    for h in hs:
        gpu_ctx.release_data(h)


def test_infinite_psd_bins(gpu_ctx, oracle):
    """A PSD of infinity takes its bin out (finite pairs); a zero PSD, whose weight is infinite, keeps the FP64
    bins: both as the oracle."""
    T, N = 8.0, 900
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    psd[100:140] = np.inf
    data = W.noise(f, 4)
    draws = W.prior_draws(4, 2)
    ref = np.array([oracle.loglik(oracle.params_from_dict(x), f, ["Hanford"], [data], [psd], T_segment=T) for x in draws])
    h = gpu_ctx.register_data("Hanford", f, data, psd)
    psd0 = psd.copy()
    psd0[N - 1] = 0.0
    h0 = gpu_ctx.register_data("Hanford", f, data, psd0)
    try:
        out, st = gpu_ctx.loglik_batch(G.params_array(draws), 0, [h], T, G.PREC_FP64)
        assert np.all(st == 0) and _close(out, ref)
        out, st = gpu_ctx.loglik_batch(G.params_array(draws), 0, [h0], T, G.PREC_FP64)
        assert np.all(st == 0) and not np.any(np.isfinite(out))
    finally:
        gpu_ctx.release_data(h)
        gpu_ctx.release_data(h0)


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_MIXED])
def test_prologue_block_sizes(gpu_ctx, prec):
    """2, 4, 8 or 16 requests per prologue block (by the number of requests): each request as in a small batch, to
    the bit in the mixed form (the FP64 form's tile, and with it its order of summation, follows the batch)."""
    T = 4.0
    f = 20.0 + np.arange(300) / T
    psd = W.analytic_psd(f)
    hs = [gpu_ctx.register_data(d, f, W.noise(f, 60 + i), psd) for i, d in enumerate(DETS[:2])]
    try:
        n = 1219
        draws = [x for pair in zip(W.prior_draws(610, 5), W.prior_draws(610, 6, precessing=True)) for x in pair][:n]
        aps = np.arange(n, dtype=np.int32) % 2
        few = np.concatenate([gpu_ctx.loglik_batch(G.params_array(draws[i:i + 100]), aps[i:i + 100], hs, T, prec)[0]
                              for i in range(0, n, 100)])
        for m in (1, 3, 304, 305, 608, 609, 1216, 1217, n):
            out, st = gpu_ctx.loglik_batch(G.params_array(draws[:m]), aps[:m], hs, T, prec)
            assert np.all(st == 0)
            if prec == G.PREC_MIXED:
                assert np.array_equal(out, few[:m])
            else:
                assert np.all(np.abs(out - few[:m]) <= 1e-11 * np.maximum(1.0, np.abs(few[:m])))
    finally:
        for h in hs:
            gpu_ctx.release_data(h)


@pytest.mark.parametrize("T,N,ndet", [(8, 90, 1), (8, 2047, 2), (4, 2048, 1), (8, 2049, 4), (12, 5003, 3)])
@pytest.mark.parametrize("ap", [0, 1])
def test_maximized(gpu_ctx, oracle, T, N, ndet, ap):
    """The maximised likelihood's two-float bins at tile edges, odd lengths and a rounded grid."""
    f, data, psd, hs = _network(gpu_ctx, oracle, T, N, ndet)
    try:
        draws = [W.config1_source(), dict(W.config1_source(), spin1=(0.3, 0.1, 0.2))] + W.prior_draws(3, N, precessing=bool(ap))
        bad = dict(draws[0], mass1=-3.0)
        ref = np.array([oracle.maximized_loglik_intrinsic(d, f, data, psd, approximant=ap) for d in draws])
        out, st = gpu_ctx.maximized_loglik_batch(G.params_array(draws + [bad]), hs, ap)
        assert np.all(st[:-1] == 0) and st[-1] != 0 and np.isnan(out[-1])
        assert _close(out[:-1], ref), np.abs(out[:-1] - ref)
    finally:
        for h in hs:
            gpu_ctx.release_data(h)


@pytest.mark.parametrize("T,N,ndet,same", [(8, 2, 1, True), (8, 127, 2, False), (1, 2047, 3, True), (1, 2049, 4, False),
                                           (8, 8113, 3, True)])
@pytest.mark.parametrize("order,eps,mode", [(2, 1e-6, 1), (4, 1e-8, 0), (2, 3e-4, 1)])
def test_fisher_moments(gpu_ctx, T, N, ndet, same, order, eps, mode):
    """The two-float moment sums against the FP64 ones on the same coefficients
    (a call with a source that two floats cannot hold, a ringdown beyond 2^24
    bins, takes FP64 sums): every region, boundary bins and cuts inside the grid,
    equal masses, steps beyond the series.  A bin's phase difference is a sum of
    at most 14 products with 2^-47 of the largest each, whose largest exceeds the
    sum by less than 100: below 1e-11."""
    f = (np.arange(N) + 10 * T) / T
    psd = W.analytic_psd(f)
    hs = [gpu_ctx.register_data(d, f, np.zeros(f.size, complex), psd if same else psd * (1 + 0.3 * i + f / 500.0))
          for i, d in enumerate(DETS[:ndet])]
    draws = W.prior_draws(9, 91)
    draws += [dict(draws[0], mass1=30.0, mass2=30.0 * (1 - 1e-5)), dict(draws[1], mass1=20.0, mass2=20.0),
              dict(draws[2], mass1=300.0, mass2=200.0), dict(draws[3], mass1=1.6, mass2=1.2)]
    kw = dict(order=order, epsilon=eps, step_mode=mode, precision=G.PREC_FP64, algorithm=G.FISHER_MOMENTS,
              covariance=False)
    got, _, st = gpu_ctx.fisher_batch_ex(G.params_array(draws), 1, hs, **kw)
    ref, _, sr = gpu_ctx.fisher_batch_ex(G.params_array(draws + [dict(draws[3], mass1=2e-6, mass2=1e-6)]), 1, hs, **kw)
    assert np.array_equal(st, sr[:-1]) and np.all(st == 0)
    assert N < 100 or np.any(got != ref[:-1])
    for i, d in enumerate(draws):
        s = np.sqrt(np.maximum(np.diag(ref[i]), 1e-300))
        assert np.max(np.abs(got[i] - ref[i]) / np.outer(s, s)) <= 1e-11, (i, d)
    for h in hs:
        gpu_ctx.release_data(h)


@pytest.mark.parametrize("N,ndet,log10F", [(2, 1, False), (255, 2, False), (257, 3, True), (1537, 4, False), (3001, 3, False)])
@pytest.mark.parametrize("ap", [0, 1])
def test_nodes(gpu_ctx, oracle, N, ndet, log10F, ap):
    """Grids that are not uniform: Gauss-Chebyshev nodes in frequency or its logarithm, in any order,
    reaching beyond the cut, in one batch with a uniform grid; the coarsest and finest node spacing, a
    source with the cut inside the grid, and one whose phase falls back to FP64."""
    th = np.pi * (np.arange(N) + 0.5) / N
    x, w = -np.cos(th), np.pi / N * np.sin(th)
    lo, hi = (np.log10(12.0), np.log10(1900.0)) if log10F else (12.0, 1900.0)
    f, w = lo + 0.5 * (hi - lo) * (x + 1), 0.5 * (hi - lo) * w
    f = 10.0 ** f if log10F else f
    perm = np.random.default_rng(N).permutation(N)
    f, w = np.ascontiguousarray(f[perm]), np.ascontiguousarray(w[perm])
    psd = [W.analytic_psd(f) * (1.0 if ndet == 3 else 1 + 0.3 * i) for i in range(ndet)]
    rng = np.random.default_rng(3)
    data = [np.sqrt(4.0 * q) * (rng.standard_normal(N) + 1j * rng.standard_normal(N)) for q in psd]
    hs = [gpu_ctx.register_data(d, f, data[i], psd[i], weights=w, log10F=log10F) for i, d in enumerate(DETS[:ndet])]
    T = 16.0
    _, udata, upsd, uh = _network(gpu_ctx, oracle, 16, 300, ndet)
    uf = 20.0 + np.arange(300) / 16.0
    src = W.config1_source()
    draws = W.prior_draws(6, 40 + N, precessing=bool(ap)) + [src, dict(src, mass1=150.0, mass2=90.0),
                                                             dict(src, mass1=70.0, mass2=1.2)]
    p = [oracle.params_from_dict(d) for d in draws]
    ref = np.array([oracle.loglik_gl(q, f, DETS[:ndet], data, psd, [w] * ndet, log10F=log10F, approximant=ap,
                                     T_segment=T) for q in p])
    out, st = gpu_ctx.loglik_batch(G.params_array(draws), ap, hs, T, G.PREC_FP64)
    assert np.all(st == 0) and _close(out, ref)
    mix, st = gpu_ctx.loglik_batch(G.params_array(draws + draws), ap, np.array([hs] * len(draws) + [uh] * len(draws)), T,
                                   G.PREC_FP64)
    uni, _ = gpu_ctx.loglik_batch(G.params_array(draws), ap, uh, T, G.PREC_FP64)
    assert np.all(st == 0) and _close(mix[:len(draws)], ref) and _close(mix[len(draws):], uni)
    for h in hs + uh:
        gpu_ctx.release_data(h)


def test_offset_and_odd_grids(gpu_ctx, oracle):
    """Simpson's rule on a uniform grid that starts between multiples of its spacing (nodes), and grids
    that keep the FP64 bins: a zero frequency."""
    f = 20.03 + np.arange(1500) / 8.0
    psd, data = W.analytic_psd(f), W.noise(f, 4)
    draws = W.prior_draws(5, 12)
    h = gpu_ctx.register_data("Virgo", f, data, psd)
    ref = np.array([oracle.loglik(oracle.params_from_dict(d), f, ["Virgo"], [data], [psd], T_segment=8.0) for d in draws])
    out, st = gpu_ctx.loglik_batch(G.params_array(draws), 0, [h], 8.0, G.PREC_FP64)
    gpu_ctx.release_data(h)
    assert np.all(st == 0) and _close(out, ref)
    f = np.concatenate([[0.0], 30.0 + np.sort(np.random.default_rng(1).uniform(0, 100, 99))])
    h = gpu_ctx.register_data("Virgo", f, np.zeros(100, complex), W.analytic_psd(f + 1), weights=np.ones(100))
    out, st = gpu_ctx.loglik_batch(G.params_array(draws), 0, [h], 8.0, G.PREC_FP64)
    gpu_ctx.release_data(h)
    assert np.all(st == 0) and out.shape == (5,)


@pytest.mark.parametrize("N", [4099, 8191, 8209, 16411, 32771, 65537, 131101])
@pytest.mark.parametrize("ap", [0, 1])
def test_maximized_transform_lengths(gpu_ctx, oracle, N, ap):
    """Every padded length of the row convolution (2^14 .. 2^18, and one on each side), the grid mostly
    just beyond a power of two: the maximum over the lags against the oracle's FP64 transform."""
    T = max(4, N // 1500)
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    data = [W.noise(f, 6 + i) for i in range(2)]
    hs = [gpu_ctx.register_data(d, f, data[i], psd) for i, d in enumerate(DETS[:2])]
    draws = W.prior_draws(3, N, precessing=bool(ap))
    ref = np.array([oracle.maximized_loglik_intrinsic(d, f, data, [psd] * 2, approximant=ap) for d in draws])
    out, st = gpu_ctx.maximized_loglik_batch(G.params_array(draws), hs, ap)
    for h in hs:
        gpu_ctx.release_data(h)
    assert np.all(st == 0) and _close(out, ref)

"""The one-request FP64 calls on node arrays (quadrature nodes, uniform grids off the line), at the edges of blocks,
against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
DETS = ("Hanford", "Livingston", "Virgo", "Kagra")


@pytest.mark.parametrize("N,ndet", [(2, 1), (127, 2), (128, 4), (129, 3), (1025, 3)])
@pytest.mark.parametrize("kind", ["quadrature", "offset"])
@pytest.mark.parametrize("ap", [0, 1])
def test_plain(gpu_ctx, oracle, N, ndet, kind, ap):
    T = 16.0
    if kind == "quadrature":
        th = np.pi * (np.arange(N) + 0.5) / N
        f, w = 12.0 + 0.5 * 1888.0 * (1 - np.cos(th)), 944.0 * np.pi / N * np.sin(th)
        perm = np.random.default_rng(N).permutation(N)
        f, w = np.ascontiguousarray(f[perm]), np.ascontiguousarray(w[perm])
    else:
        f, w = 20.0 + 3e-8 + np.arange(N) / T, None
    psd = [W.analytic_psd(f) * (1.0 if ndet == 3 else 1 + 0.3 * i) for i in range(ndet)]
    rng = np.random.default_rng(3)
    data = [np.sqrt(4.0 * q) * (rng.standard_normal(N) + 1j * rng.standard_normal(N)) for q in psd]
    hs = [gpu_ctx.register_data(d, f, data[i], psd[i], weights=w) for i, d in enumerate(DETS[:ndet])]
    src = W.config1_source()
    method = "IMRPhenomPv2" if ap else "IMRPhenomD"
    cell = torch.zeros(1, dtype=torch.float64, device="cuda")
    try:
        for d in W.prior_draws(4, N, precessing=bool(ap)) + [src, dict(src, mass1=150.0, mass2=90.0),
                                                            dict(src, mass1=70.0, mass2=1.2)]:
            p = oracle.params_from_dict(d)
            if w is None:
                ref = oracle.loglik(p, f, list(DETS[:ndet]), data, psd, approximant=ap, T_segment=T)
            else:
                ref = oracle.loglik_gl(p, f, DETS[:ndet], data, psd, [w] * ndet, approximant=ap, T_segment=T)
            got = gpu_ctx.mcmc_likelihood_extrinsic(G.gen_params(**d), method, hs, T)
            assert abs(got - ref) <= 1e-9 * max(1.0, abs(ref)), (d, got, ref)
            st = gpu_ctx.lib.gwgpu_mcmc_likelihood_extrinsic_noalloc(
                gpu_ctx.h, ctypes.byref(G.gen_params(**d)), method.encode(), (ctypes.c_int * ndet)(*hs), ndet, T,
                ctypes.c_void_p(cell.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0 and cell.item() == got
    finally:
        for h in hs:
            gpu_ctx.release_data(h)

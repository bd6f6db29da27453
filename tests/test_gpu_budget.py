"""A context with a device-memory budget: the FP64 form's two-float arrays, which a registration takes while there
is room, give way to whatever needs it later."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu
T, N = 16.0, 16001
DETS = ("Hanford", "Livingston")
ENTRIES = 65537  # of the tables by bin


def _batch(prec, n):
    def call(ctx, hs):
        return ctx.loglik_batch(G.params_array(W.prior_draws(n, 3)), 0, hs, T, prec)[0]
    return call


def _maximized(ap):
    def call(ctx, hs):
        return ctx.maximized_loglik_batch(G.params_array(W.prior_draws(8, 3, precessing=bool(ap))), hs, ap)[0]
    return call


def _fisher(n):
    def call(ctx, hs):
        return ctx.fisher_batch_ex(G.params_array(W.prior_draws(n, 3)), 1, hs, order=2, epsilon=1e-6, step_mode=1,
                                   precision=G.PREC_FP64, algorithm=G.FISHER_MOMENTS, covariance=False)[0]
    return call


def _another(ctx, hs):
    f = 20.0 + np.arange(2 * N) / T
    h = [ctx.register_data(d, f, W.noise(f, 7), W.analytic_psd(f)) for d in DETS]
    return ctx.loglik_batch(G.params_array(W.prior_draws(4, 3)), 0, h, T, G.PREC_FP64)[0]


def _plain(ctx, hs):
    f = 20.0 + np.arange(500000) / 1024.0
    ctx.register_data("Virgo", f, W.noise(f, 7), W.analytic_psd(f))
    p = [G.gen_params(**d) for d in W.prior_draws(4, 3)]
    return np.array([ctx.mcmc_likelihood_extrinsic(x, "IMRPhenomD", hs, T) for x in p])


@pytest.mark.parametrize("grid", ["bins", "nodes"])
@pytest.mark.parametrize("name,call", [("mixed", _batch(G.PREC_MIXED, 3000)), ("fp64", _batch(G.PREC_FP64, 3000)),
                                       ("maximized", _maximized(0)), ("maximized unaligned", _maximized(1)),
                                       ("fisher", _fisher(64)), ("registration", _another), ("plain", _plain)])
def test_two_float_arrays_give_way(name, call, grid):
    """A budget that holds all but half of them, or none."""
    if grid == "nodes" and name in ("mixed", "maximized", "maximized unaligned", "fisher"):
        f = 20.0 + 1e-8 + np.arange(N) / T  # uniform for these calls, nodes for the FP64 form
    elif grid == "nodes":
        f = 20.3 / T + 20.0 + np.arange(N) / T
    else:
        f = 20.0 + np.arange(N) / T
    psd, data = W.analytic_psd(f), [W.noise(f, 4 + i) for i in range(2)]

    def run(budget, data=data):
        ctx = G.Context(0, hbm_budget=budget)
        try:
            hs = [ctx.register_data(d, f, data[i], psd) for i, d in enumerate(DETS)]
            before = ctx.loglik_batch(G.params_array(W.prior_draws(5, 6)), 0, hs, T, G.PREC_FP64)[0]
            out = call(ctx, hs)
            used = ctx.bytes_in_use()
            # and what was asked before is answered as before
            after = ctx.loglik_batch(G.params_array(W.prior_draws(5, 6)), 0, hs, T, G.PREC_FP64)[0]
            close = np.abs(after - before) <= 1e-9 * np.maximum(1.0, np.abs(before))
            assert np.all(close | np.isnan(before))
            return out, used
        finally:
            ctx.close()

    ref, used = run(0)
    extra = 2 * 28 * N + 80 * ENTRIES if grid == "bins" else 2 * 120 * N
    budget = used - extra // 2
    if name == "fp64":  # what the call takes on streams that never had them: its plan is another
        budget = run(0, [np.where(np.arange(N) == N - 1, np.nan, d) for d in data])[1]
    got, less = run(budget)
    assert less <= budget
    if name == "fisher":
        s = np.sqrt(np.einsum("nii->ni", ref))
        assert np.max(np.abs(got - ref) / (s[:, :, None] * s[:, None, :])) <= 1e-11
    else:
        assert np.all(np.abs(got - ref) <= (1e-6 if name == "mixed" else 1e-9) * np.maximum(1.0, np.abs(ref)))


def test_a_budget_that_suffices_keeps_them():
    f = 20.0 + np.arange(N) / T
    psd, data = W.analytic_psd(f), W.noise(f, 4)
    p = G.params_array(W.prior_draws(50, 6))
    outs, used = [], 0
    for _ in range(2):
        ctx = G.Context(0, hbm_budget=used)
        h = ctx.register_data("Virgo", f, data, psd)
        outs.append(ctx.loglik_batch(p, 0, [h], T, G.PREC_FP64)[0])
        used = ctx.bytes_in_use()
        ctx.close()
    assert np.array_equal(*outs)


def test_a_captured_call_keeps_them():
    """A call without allocation, captured by the caller: what it reads stays, and what needs its place is refused."""
    import ctypes

    import torch
    f = 20.0 + np.arange(N) / T
    psd, data = W.analytic_psd(f), W.noise(f, 4)

    def run(budget, capture):
        ctx = G.Context(0, hbm_budget=budget)
        try:
            h = (ctypes.c_int * 1)(ctx.register_data("Virgo", f, data, psd))
            p = G.gen_params(**W.prior_draws(1, 6)[0])
            cell = torch.zeros(1, dtype=torch.float64, device="cuda")

            def call(stream):
                assert ctx.lib.gwgpu_mcmc_likelihood_extrinsic_noalloc(ctx.h, ctypes.byref(p), b"IMRPhenomD", h, 1, T,
                                                                       ctypes.c_void_p(cell.data_ptr()),
                                                                       ctypes.c_void_p(stream.cuda_stream)) == 0
            call(torch.cuda.current_stream())
            torch.cuda.synchronize()
            first = cell.item()
            graph = torch.cuda.CUDAGraph()
            if capture:
                with torch.cuda.graph(graph):
                    call(torch.cuda.current_stream())
            try:
                _batch(G.PREC_MIXED, 3000)(ctx, list(h))
                refused = False
            except G.engine.GwGpuError:
                refused = True
            used = ctx.bytes_in_use()
            if capture:
                cell.zero_()
                graph.replay()
                torch.cuda.synchronize()
                assert cell.item() == first
                del graph
            return used, refused
        finally:
            ctx.close()

    used, refused = run(0, False)
    assert not refused
    assert run(used - 40 * ENTRIES, False)[1] is False
    assert run(used - 40 * ENTRIES, True)[1] is True

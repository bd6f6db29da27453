"""What the framework is measured on: log-likelihood, maximised likelihood and
Fisher calls through gw_analysis_tools_gb300's Python entry points.

A case is one call that a sampler or an analysis script makes:

  plain      one request per call in FP64, the drop-in under an existing sampler
             (Context.mcmc_likelihood_extrinsic); latency counts
  batch      many requests in one call (Context.loglik_batch), mixed precision
             or FP64, IMRPhenomD or IMRPhenomPv2, on one grid, on several grids
             at once ("uneven") or on Gauss-Legendre nodes ("gaussleg")
  chains     a few chains' sampler vectors in one call (Context.mcmc_loglik_batch)
  maximized  the likelihood maximised over arrival time and phase for a batch of
             intrinsic draws (Context.maximized_loglik_batch)
  fisher     the sampler's Fisher proposal at many positions (Context.mcmc_fisher_batch)

The request server is not among them: it runs on a clock of its own, and its
device work is that of the batch cases.  Every call takes host arrays and
returns host arrays, as a sampler's does.

Inputs are synthetic: an analytic PSD, seeded Gaussian noise plus the signal of
one source, parameters drawn from the priors (batches) or around the source
(chains, plain and Fisher calls, as a converged sampler asks for).
"""
import functools
import os
import re

import numpy as np
import torch

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

DETECTORS = ("Hanford", "Livingston", "Virgo")
UNEVEN_T = (4, 8, 32, 128)
F_LOW = 20


def listed():
    return [
        # smallest call: one detector, short segment, narrow band; launch latency
        dict(name="plain_d_short", kind="plain", model="D", dets=1, T=4, fmax=512),
        # the drop-in call on the three-detector network, 32 s segment (32,128 bins)
        dict(name="plain_d", kind="plain", model="D", dets=3, T=32, fmax=1024),
        # the same for a precessing source, wider band
        dict(name="plain_pv2", kind="plain", model="P", dets=3, T=8, fmax=2048),
        # one ensemble's temperatures in one step: too few requests to fill the chip
        dict(name="chains_mixed_d", kind="chains", model="D", dets=3, T=32, fmax=1024, requests=16),
        # the parallel-tempered step: 64 chains x 8 temperatures
        dict(name="batch_mixed_d", kind="batch", prec="mixed", model="D", dets=3, T=32, fmax=1024, requests=512),
        # several analyses at once: grids of 4 to 128 s in one launch, precessing
        dict(name="uneven_mixed_pv2", kind="batch", prec="mixed", model="P", dets=3, T=0, fmax=2048, requests=1024),
        # the FP64 form of the step: checks and final evaluations
        dict(name="batch_fp64_d", kind="batch", prec="fp64", model="D", dets=3, T=32, fmax=1024, requests=512),
        # precessing requests in FP64, two detectors
        dict(name="batch_fp64_pv2", kind="batch", prec="fp64", model="P", dets=2, T=16, fmax=2048, requests=64),
        # Gauss-Legendre nodes instead of a uniform grid
        dict(name="gaussleg_fp64_d", kind="batch", prec="gaussleg", model="D", dets=3, T=32, fmax=1024, nodes=3000,
             requests=512),
        # intrinsic draws maximised over time and phase (a prime factor in the length)
        dict(name="maximized_d", kind="maximized", model="D", dets=3, T=32, fmax=1024, requests=128),
        # the precessing form on an odd grid length
        dict(name="maximized_pv2", kind="maximized", model="P", dets=3, T=16, fmax=1000, requests=48),
        # Fisher proposals for a set of chains
        dict(name="fisher_proposal", kind="fisher", model="D", dets=3, T=32, fmax=1039, requests=256),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(a * (b / a) ** rng.random()))

    kind = rng.choice(["plain", "plain", "chains", "mixed", "mixed", "uneven", "fp64", "fp64", "gaussleg", "maximized",
                       "fisher"])
    model = rng.choice(["D", "D", "P"])
    dets = rng.choice([1, 2, 3, 3])
    T = rng.choice([4, 5, 8, 12, 16, 25, 32, 50, 64])
    fmax = rng.randrange(480, 2049)
    c = dict(model=model, dets=dets, T=T, fmax=fmax)
    bins = T * (fmax - F_LOW)

    def most(total, cap, floor=1):  # requests within the work of the largest listed case of the kind
        return log_int(floor, max(floor, min(cap, total // bins)))

    if kind == "plain":
        return dict(c, kind="plain")
    if kind == "chains":
        return dict(c, kind="chains", requests=log_int(1, 64))
    if kind == "mixed":
        return dict(c, kind="batch", prec="mixed", requests=most(16_000_000, 1024, 4))
    if kind == "uneven":
        return dict(c, kind="batch", prec="mixed", T=0, requests=log_int(16, 1000))
    if kind == "fp64":
        return dict(c, kind="batch", prec="fp64", requests=most(8_000_000 if model == "D" else 2_000_000, 512, 2))
    if kind == "gaussleg":
        return dict(c, kind="batch", prec="gaussleg", model="D", nodes=log_int(200, 4000), requests=log_int(8, 384))
    if kind == "maximized":
        c.update(T=min(T, 32), fmax=min(fmax, 1100))
        bins = c["T"] * (c["fmax"] - F_LOW)
        return dict(c, kind="maximized", requests=max(2, min(128, log_int(200_000, 3_000_000 if model == "D" else 700_000) // bins)))
    c.update(model="D", T=min(T, 32), fmax=min(fmax, 1040))
    return dict(c, kind="fisher", requests=log_int(4, 256))


# ------------------------------------------------------------------ inputs
def grids(case):
    """[(T, frequencies, integration weights or None)]: one, or one per segment length."""
    if case.get("prec") == "gaussleg":
        x, w = gauss_legendre(case["nodes"])
        half = 0.5 * (case["fmax"] - F_LOW)
        return [(case["T"], F_LOW + half * (x + 1.0), half * w)]
    return [(T, F_LOW + np.arange(T * (case["fmax"] - F_LOW)) * (1.0 / T), None)
            for T in (UNEVEN_T if case["T"] == 0 else (case["T"],))]


@functools.lru_cache(maxsize=8)
def gauss_legendre(n):
    x = np.cos(np.pi * (np.arange(n, 0, -1) - 0.25) / (n + 0.5))
    for _ in range(6):  # Newton on P_n by its recurrence
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        dp = n * (x * p1 - p0) / (x * x - 1.0)
        x = x - p1 / dp
    return x, 2.0 / ((1.0 - x * x) * dp * dp)


def source(model):
    s = dict(W.config1_source(), tc=0.02)
    if model == "P":
        s.update(spin1=(0.25, -0.1, 0.3), spin2=(-0.1, 0.2, -0.1))
    return s


def parameters(case, seed):
    """The parameter dicts of a case's requests."""
    pre = case["model"] == "P"
    if case["kind"] in ("batch", "maximized"):
        return W.prior_draws(case["requests"], seed, precessing=pre)
    return W.perturbed(source(case["model"]), case.get("requests", 1), seed)


def vectors(plist, model):
    """Sampler vectors: RA, sin DEC, psi, cos iota, phiRef, tc, ln D_L, ln M_c, eta, then the
    aligned spins, or magnitudes, cosines of the tilts and azimuths."""
    out = []
    for p in plist:
        m1, m2 = p["mass1"], p["mass2"]
        v = [p["RA"], np.sin(p["DEC"]), p["psi"], np.cos(p["incl_angle"]), p["phiRef"], p["tc"],
             np.log(p["Luminosity_Distance"]), np.log((m1 * m2) ** 0.6 / (m1 + m2) ** 0.2), m1 * m2 / (m1 + m2) ** 2]
        s1, s2 = np.array(p["spin1"]), np.array(p["spin2"])
        if model == "P":
            a1, a2 = np.linalg.norm(s1), np.linalg.norm(s2)
            v += [a1, a2, s1[2] / a1, s2[2] / a2, np.arctan2(s1[1], s1[0]), np.arctan2(s2[1], s2[0])]
        else:
            v += [s1[2], s2[2]]
        out.append(v)
    return np.array(out)


def streams(case, seed):
    """[(T, f, weights, psd, [data per detector])] and each request's grid."""
    src = source(case["model"])
    out = []
    for g, (T, f, w) in enumerate(grids(case)):
        psd = W.analytic_psd(f)
        ft = torch.from_numpy(f).cuda()
        sig = responses(dict(src, tc=T - src["tc"]), case["model"], ft, case["dets"])
        rng = np.random.Generator(np.random.PCG64([seed, g]))
        sd = np.sqrt(psd * T / 4.0)
        data = [s.cpu().numpy() + sd * (rng.standard_normal(f.size) + 1j * rng.standard_normal(f.size)) for s in sig]
        out.append((T, f, w, psd, data))
    n = case.get("requests", 1)
    which = np.random.Generator(np.random.PCG64(seed)).integers(0, len(out), n) if len(out) > 1 else np.zeros(n, int)
    return out, which


def prepare(case, seed):
    ctx = G.Context(0)
    data, which = streams(case, seed)
    handles = [[ctx.register_data(DETECTORS[d], f, dat[d], psd, weights=w) for d in range(case["dets"])]
               for (_, f, w, psd, dat) in data]
    plist = parameters(case, seed + 1)
    state = dict(ctx=ctx, case=case, T=float(data[0][0]))
    # T <= 0: every request's t_c counts from the end of its own segment
    if len(data) > 1:
        state.update(T=0.0, handles=np.array([handles[g] for g in which], dtype=np.int32))
    else:
        state.update(handles=handles[0])
    state["approx"] = G.IMRPhenomPv2 if case["model"] == "P" else G.IMRPhenomD
    if case["kind"] in ("chains", "fisher"):
        state["theta"] = vectors(plist, case["model"])
    else:
        state["params"] = G.params_array(plist)
    if case["kind"] == "plain":
        state["method"] = "IMRPhenomPv2" if case["model"] == "P" else "IMRPhenomD"
    if case["kind"] == "batch":
        state["prec"] = G.PREC_MIXED if case["prec"] == "mixed" else G.PREC_FP64
    return state


def run(s):
    kind, ctx = s["case"]["kind"], s["ctx"]
    if kind == "plain":
        return np.array([ctx.mcmc_likelihood_extrinsic(s["params"][0], s["method"], s["handles"], s["T"])])
    if kind == "batch":
        return ctx.loglik_batch(s["params"], s["approx"], s["handles"], s["T"], precision=s["prec"])
    if kind == "chains":
        return ctx.mcmc_loglik_batch(s["theta"], s["approx"], W.GMST, s["handles"], s["T"], precision=G.PREC_MIXED)
    if kind == "maximized":
        return ctx.maximized_loglik_batch(s["params"], s["handles"], s["approx"])
    return ctx.mcmc_fisher_batch(s["theta"], s["handles"], W.GMST)


def work(case):
    """Data, PSD and frequencies once, parameters and results once; operations of the
    reference algorithm: 67 (IMRPhenomD) or 239 (IMRPhenomPv2) a waveform bin, 33 a detector
    bin, per request; a Fisher takes the waveform at 44 perturbed parameter sets (order 4)
    and 66 products a detector bin; a maximised request adds a transform per detector (and
    polarisation)."""
    n, dets = case.get("requests", 1), case["dets"]
    sizes = [f.size for _, f, _ in grids(case)]
    per_bin = (67.0 if case["model"] == "D" else 239.0) + 33.0 * dets
    flops = n * per_bin * sum(sizes) / len(sizes)
    nbytes = 32.0 * dets * sum(sizes) + n * (176 + 12)
    if case["kind"] == "fisher":
        flops = n * sizes[0] * (44.0 * (67 + 12 * dets) + 66 * 4 * dets)
        nbytes += n * 11 * 11 * 8
    if case["kind"] == "maximized":
        flops += n * dets * (1 if case["model"] == "D" else 2) * 5.0 * sizes[0] * np.log2(sizes[0])
    return {"bytes": float(nbytes), "flops": float(flops)}


# --------------------------------------------------- the same in plain torch
# IMRPhenomD (arXiv:1508.07253) and IMRPhenomPv2 (arXiv:1308.3271) with the conventions of
# gw_analysis_tools, written for 64-bit tensors.  Only the calibrated numbers come from the
# package: its table of fits, quasi-normal frequencies and detectors.
MSUN, MPC, C = 4.925491025543575903411922162094833998e-6, 3.085677581491367278913937957796471611e22, 299792458.0
PI = np.pi
EULER_GAMMA, LOG64 = 0.5772156649015328606, 4.15888308336


@functools.lru_cache(maxsize=1)
def tables():
    with open(os.path.join(os.path.dirname(G.__file__), "csrc", "phenom_tables.h")) as f:
        text = f.read()

    def numbers(name):
        body = re.search(r"#define GWT_%s_INIT (.*?)\n(?:static|#)" % name, text, re.S).group(1)
        return np.array([float(x) for x in re.findall(r"[-+]?\d+\.?\d*(?:[eE][-+]?\d+)?", body)])

    a, ring, damp = numbers("QNM_A"), numbers("QNM_FRING"), numbers("QNM_FDAMP")
    return dict(fits=numbers("LAMBDA_FIT").reshape(19, 11), a=a, ring=(ring, spline(a, ring)), damp=(damp, spline(a, damp)),
                loc=numbers("DET_LOCATION").reshape(9, 3), tensor=numbers("DET_TENSOR").reshape(9, 3, 3),
                geom=numbers("DET_GEOMETRIC"))


def spline(x, y):
    """Second derivatives of the natural cubic spline through (x, y)."""
    n, h = x.size, np.diff(x)
    A, b = np.eye(n), np.zeros(n)
    s = np.diff(y) / h
    for i in range(1, n - 1):
        A[i, i - 1:i + 2] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        b[i] = 6 * (s[i] - s[i - 1])
    return np.linalg.solve(A, b)


def spline_at(x, y, m, v, slope=False):
    i = int(np.clip(np.searchsorted(x, v, side="right") - 1, 0, x.size - 2))
    h, a, b = x[i + 1] - x[i], x[i + 1] - v, v - x[i]
    if slope:
        return ((y[i + 1] - y[i]) / h - h * (m[i + 1] - m[i]) / 6 + (m[i + 1] * b * b - m[i] * a * a) / (2 * h))
    return ((m[i] * a ** 3 + m[i + 1] * b ** 3) / (6 * h) + (y[i] / h - m[i] * h / 6) * a + (y[i + 1] / h - m[i + 1] * h / 6) * b)


def final_spin(eta, chi1, chi2):
    d = np.sqrt(max(0.0, 1 - 4 * eta))
    s = ((1 + d) / 2) ** 2 * chi1 + ((1 - d) / 2) ** 2 * chi2
    return eta * (3.4641016151377544 - 4.399247300629289 * eta + 9.397292189321194 * eta ** 2 - 13.180949901606242 * eta ** 3
                  + s * (1 / eta - 0.0850917821418767 - 5.837029316602263 * eta)
                  + s ** 2 * (0.1014665242971878 - 2.0967746996832157 * eta)
                  + s ** 3 * (-1.3546806617824356 + 4.108962025369336 * eta)
                  + s ** 4 * (-0.8676969352555539 + 2.064046835273906 * eta))


def radiated(eta, chi1, chi2):
    d = np.sqrt(max(0.0, 1 - 4 * eta))
    w1, w2 = ((1 + d) / 2) ** 2, ((1 - d) / 2) ** 2
    s = (w1 * chi1 + w2 * chi2) / (w1 + w2)
    num = 1 + s * (-0.0030302335878845507 - 2.0066110851351073 * eta + 7.7050567802399215 * eta ** 2)
    den = 1 + s * (-0.6714403054720589 - 1.4756929437702908 * eta + 7.304676214885011 * eta ** 2)
    return eta * (0.055974469826360077 + 0.5809510763115132 * eta - 0.9606726679372312 * eta ** 2 + 3.352411249771192 * eta ** 3) * num / den


class PhenomD:
    """The constants of one source in units of x = M f, and its amplitude and phase."""

    def __init__(self, p, spin_in_plane=None):
        m1, m2 = p["mass1"] * MSUN, p["mass2"] * MSUN
        c1, c2 = p["spin1"][2], p["spin2"][2]
        self.m1, self.m2 = m1, m2
        M = self.M = m1 + m2
        eta = self.eta = m1 * m2 / (M * M)
        cs, ca, dm = (c1 + c2) / 2, (c1 - c2) / 2, np.sqrt(max(0.0, 1 - 4 * eta))
        chi_pn = (m1 * c1 + m2 * c2) / M - 38.0 / 113 * eta * 2 * cs
        mc, dl = M * eta ** 0.6, p["Luminosity_Distance"] * MPC / C
        self.A0 = np.sqrt(PI * 40.0 / 192) * mc * mc / dl * (PI * mc) ** (-7.0 / 6)
        t = tables()
        xi = chi_pn - 1
        e = np.array([1, eta, eta * eta])
        fits = t["fits"]
        lam = fits[:, 0] + fits[:, 1] * eta + sum(xi ** (k + 1) * (fits[:, 2 + 3 * k:5 + 3 * k] @ e) for k in range(3))
        self.rho, v2, self.gam, self.sig, self.bet, self.alp = lam[0:3], lam[3], lam[4:7], lam[7:11], lam[11:14], lam[14:19]
        af = final_spin(eta, c1, c2)
        if spin_in_plane is not None:
            af = np.copysign(1.0, af) * np.hypot(spin_in_plane * (max(m1, m2) / M) ** 2, af)
        er = radiated(eta, c1, c2)
        self.xr = spline_at(t["a"], *t["ring"], af) / (1 - er)
        self.xd = spline_at(t["a"], *t["damp"], af) / (1 - er)
        # post-Newtonian amplitude and phase coefficients of (pi x)^(i/3)
        e2, e3, ca2, cs2 = eta ** 2, eta ** 3, ca * ca, cs * cs
        self.pa = np.array([
            1, 0, -323 / 224 + 451 / 168 * eta, 27 / 8 * dm * ca + (27 / 8 - 11 / 6 * eta) * cs,
            -27312085 / 8128512 - 1975055 / 338688 * eta + 105271 / 24192 * e2 + (-81 / 32 + 8 * eta) * ca2
            - 81 / 16 * dm * ca * cs + (-81 / 32 + 17 / 8 * eta) * cs2,
            -85 * PI / 64 + 85 * PI / 16 * eta + dm * (285197 / 16128 - 1579 / 4032 * eta) * ca
            + (285197 / 16128 - 15317 / 672 * eta - 2227 / 1008 * e2) * cs,
            -177520268561 / 8583708672 + (545384828789 / 5007163392 - 205 * PI ** 2 / 48) * eta - 3248849057 / 178827264 * e2
            + 34473079 / 6386688 * e3 + (1614569 / 64512 - 1873643 / 16128 * eta + 2167 / 42 * e2) * ca2
            + (31 * PI / 12 - 7 * PI / 3 * eta) * cs + (1614569 / 64512 - 61391 / 1344 * eta + 57451 / 4032 * e2) * cs2
            + dm * ca * (31 * PI / 12 + (1614569 / 32256 - 165961 / 2688 * eta) * cs)])
        p5 = (38645 * PI / 756 - 65 * PI / 9 * eta + dm * (-732985 / 2268 - 140 / 9 * eta) * ca
              + (-732985 / 2268 + 24260 / 81 * eta + 340 / 9 * e2) * cs)
        p6 = (11583231236531 / 4694215680 - 6848 * EULER_GAMMA / 21 - 640 * PI ** 2 / 3
              + (-15737765635 / 3048192 + 2255 * PI ** 2 / 12) * eta + 76055 / 1728 * e2 - 127825 / 1296 * e3
              + 2270 * PI / 3 * dm * ca + (2270 * PI / 3 - 520 * PI * eta) * cs - 6848 * LOG64 / 63)
        self.pp = np.array([
            1, 0, 3715 / 756 + 55 / 9 * eta, -16 * PI + 113 / 3 * dm * ca + (113 / 3 - 76 / 3 * eta) * cs,
            15293365 / 508032 + 27145 / 504 * eta + 3085 / 72 * e2 + (-405 / 8 + 200 * eta) * ca2 - 405 / 4 * dm * ca * cs
            + (-405 / 8 + 5 / 2 * eta) * cs2, p5, p6,
            77096675 * PI / 254016 + 378515 * PI / 1512 * eta - 74045 * PI / 756 * e2
            + dm * (-25150083775 / 3048192 + 26804935 / 6048 * eta - 1985 / 48 * e2) * ca
            + (-25150083775 / 3048192 + 10566655595 / 762048 * eta - 1042165 / 3024 * e2 + 5345 / 36 * e3) * cs])
        self.l5, self.l6 = p5, -6848 / 63  # the coefficients of ln(pi x) beside p5 and p6
        # amplitude: regions and the quartic between them
        g1, g2, g3 = self.gam
        peak = self.xr - self.xd * g3 / g2 if g2 > 1 else self.xr + self.xd * g3 * (np.sqrt(1 - g2 * g2) - 1) / g2
        self.x1, self.x3, self.cut = 0.014, abs(peak), 0.2
        x1, x3 = self.x1, self.x3
        xm, h = (x1 + x3) / 2, (x3 - x1) / 2
        w = g3 * self.xd
        u = x3 - self.xr
        v1, d1 = self._ins_amp_scalar(x1)
        v3 = g1 * w * np.exp(-g2 * u / w) / (u * u + w * w)
        d3 = v3 * (-g2 / w - 2 * u / (u * u + w * w))
        A = np.array([[(-1.0) ** k for k in range(5)], [1, 0, 0, 0, 0], [1.0] * 5,
                      [k * (-1.0) ** (k - 1) if k else 0 for k in range(5)], [float(k) for k in range(5)]])
        self.quart = np.linalg.solve(A, np.array([v1, v2, v3, d1 * h, d3 * h]))
        self.xm, self.h = xm, h
        # phase: C1 connections at 0.018 and half the ringdown frequency
        self.p1, self.p2 = 0.018, self.xr / 2
        self.a1fit = self.alp[1 - 1]
        b1, b2, b3 = self.bet
        a1, a2, a3, a4, a5 = self.alp
        ph, dph = self._ins_phase_scalar(self.p1)
        x = self.p1
        b1 = eta * dph - (b2 / x + b3 / x ** 4)
        b0 = eta * ph - (b1 * x + b2 * np.log(x) - b3 / (3 * x ** 3))
        self.beta = (b0, b1, b2, b3)
        x = self.p2
        y = (x - a5 * self.xr) / self.xd
        a1 = (b1 + b2 / x + b3 / x ** 4) - (a2 / x ** 2 + a3 / x ** 0.25 + a4 / (self.xd * (1 + y * y)))
        a0 = (b0 + b1 * x + b2 * np.log(x) - b3 / (3 * x ** 3)) - (a1 * x - a2 / x + 4 / 3 * a3 * x ** 0.75 + a4 * np.arctan(y))
        self.alpha = (a0, a1, a2, a3, a4, a5)

    def _ins_amp_scalar(self, x):
        v, y = (PI * x) ** (1 / 3), x ** (1 / 3)
        val = sum(self.pa[i] * v ** i for i in range(7)) + sum(self.rho[i] * y ** (7 + i) for i in range(3))
        der = (sum(self.pa[i] * v ** i * i for i in range(7)) + sum(self.rho[i] * y ** (7 + i) * (7 + i) for i in range(3))) / (3 * x)
        return val, der

    def _ins_phase_scalar(self, x):
        v, L = (PI * x) ** (1 / 3), np.log(PI * x)
        c = self.pp.copy()
        c[5] += self.l5 * L
        c[6] += self.l6 * L
        k = 3 / (128 * self.eta)
        s = sum(c[i] * v ** i for i in range(8))
        ds = sum(c[i] * v ** i * i for i in range(8)) / (3 * x) + (self.l5 * v ** 5 + self.l6 * v ** 6) / x
        s1, s2, s3, s4 = self.sig
        ph = -PI / 4 + k * v ** -5 * s + (s1 * x + 0.75 * s2 * x ** (4 / 3) + 0.6 * s3 * x ** (5 / 3) + 0.5 * s4 * x * x) / self.eta
        dph = k * v ** -5 * (ds - 5 / (3 * x) * s) + (s1 + s2 * x ** (1 / 3) + s3 * x ** (2 / 3) + s4 * x) / self.eta
        return ph, dph

    def amplitude(self, x):
        """Amplitude without its A0 x^(-7/6)."""
        y = x ** (1.0 / 3)
        c = [self.pa[i] * PI ** (i / 3) for i in range(7)] + list(self.rho)
        ins = torch.zeros_like(x)
        for k in reversed(c):
            ins = ins * y + k
        u = (x - self.xm) / self.h
        mid = torch.zeros_like(x)
        for k in reversed(list(self.quart)):
            mid = mid * u + k
        g1, g2, g3 = self.gam
        w = g3 * self.xd
        d = x - self.xr
        ring = g1 * w * torch.exp(-g2 * d / w) / (d * d + w * w)
        return torch.where(x < self.x1, ins, torch.where(x > self.x3, ring, mid))

    def phase(self, x):
        v, L = (PI * x) ** (1.0 / 3), torch.log(PI * x)
        s = torch.zeros_like(x)
        for i in reversed(range(8)):
            c = self.pp[i] + (self.l5 * L if i == 5 else self.l6 * L if i == 6 else 0.0)
            s = s * v + c
        s1, s2, s3, s4 = self.sig
        y = x ** (1.0 / 3)
        ins = -PI / 4 + 3 / (128 * self.eta) * s / v ** 5 + (s1 * x + 0.75 * s2 * x * y + 0.6 * s3 * x * y * y + 0.5 * s4 * x * x) / self.eta
        b0, b1, b2, b3 = self.beta
        mid = (b0 + b1 * x + b2 * torch.log(x) - b3 / (3 * x ** 3)) / self.eta
        a0, a1, a2, a3, a4, a5 = self.alpha
        ring = (a0 + a1 * x - a2 / x + 4 / 3 * a3 * x ** 0.75 + a4 * torch.atan((x - a5 * self.xr) / self.xd)) / self.eta
        return torch.where(x < self.p1, ins, torch.where(x > self.p2, ring, mid))


def scalar(fn, x):
    return float(fn(torch.tensor([x], dtype=torch.float64))[0])


def halves(a):
    """a as a sum of two numbers of 26 bits each, so that products of halves are exact."""
    c = a * 134217729.0
    h = c - (c - a)
    return h, a - h


def turn(t, f):
    """2 pi times the fraction of t f: the turns of a time shift of seconds, with no rounding of their whole part."""
    a, b = halves(torch.full_like(f, t))
    c, d = halves(f)
    p = [a * c, a * d, b * c, b * d]
    return 2 * PI * sum(x - torch.round(x) for x in reversed(p))


def wave_d(p, f):
    """h+ and hx of IMRPhenomD, t_c and the phase at f_ref as the framework's defaults set them."""
    d = PhenomD(p)
    M, fref = d.M, p["f_ref"]
    a0, a1, a2, a3, a4, a5 = d.alpha
    y = (d.x3 - a5 * d.xr) / d.xd
    shift = M / d.eta * (d.a1fit + a2 / d.x3 ** 2 + a3 / d.x3 ** 0.25 + a4 / (d.xd * (1 + y * y)))
    x = M * f
    ph = d.phase(x) - (turn(p["tc"], f - fref) + shift * (f - fref) + 2 * p["phiRef"] + scalar(d.phase, M * fref))
    amp = torch.where(x > d.cut, 0.0, d.A0 * M ** (7 / 6) * x ** (-7.0 / 6) * d.amplitude(x))
    h = torch.polar(amp.abs(), -ph) * torch.sign(amp)
    c = np.cos(p["incl_angle"])
    return h * ((1 + c * c) / 2), h * (-1j * c)


def euler_coefficients(q, chil, chip):
    """Coefficients of alpha and epsilon in w^-1, w^-2/3, w^-1/3, ln w, w^1/3 (w = pi M f)."""
    m2, m1 = q / (1 + q), 1 / (1 + q)
    d, n = m1 - m2, m1 * m2
    out = []
    for cp2 in (chip * chip, 0.0):
        cp4 = cp2 * cp2
        out.append([
            -35 / 192 - 5 * d / (64 * m2),
            -15 * d * m2 * chil / (128 * n) - 35 * m2 ** 2 * chil / (128 * n),
            -5515 / 3072 - 4555 * d / (7168 * m2) - cp2 * (15 * d * m2 ** 3 + 35 * m2 ** 4) / (128 * n ** 2) - 515 * n / 384
            - 15 * d ** 2 * n / (256 * m2 ** 2) - 175 * d * n / (256 * m2),
            -35 * PI / 48 - 5 * d * PI / (16 * m2) + 5 * d ** 2 * chil / 16 + 5 * d * m2 * chil / 3 + 2545 * m2 ** 2 * chil / 1152
            - cp2 * chil * (5 * d * m2 ** 5 / (128 * n ** 3) + 35 * m2 ** 6 / (384 * n ** 3))
            + 2035 * d * m2 * chil / (21504 * n) + 2995 * m2 ** 2 * chil / (9216 * n),
            4.318908476114694 + 27895885 * d / (2.1676032e7 * m2) - cp4 * (15 * d * m2 ** 7 + 35 * m2 ** 8) / (512 * n ** 4)
            + cp2 * (-485 * d * m2 ** 3 / (14336 * n ** 2) + 475 * m2 ** 4 / (6144 * n ** 2) + 15 * d ** 2 * m2 ** 2 / (256 * n)
                     + 145 * d * m2 ** 3 / (512 * n) + 575 * m2 ** 4 / (1536 * n)
                     + chil ** 2 * (15 * d * m2 ** 7 + 35 * m2 ** 8) / (128 * n ** 4))
            + 39695 * n / 86016 + 1615 * d ** 2 * n / (28672 * m2 ** 2) - 265 * d * n / (14336 * m2) + 955 * n ** 2 / 576
            + 15 * d ** 3 * n ** 2 / (1024 * m2 ** 3) + 35 * d ** 2 * n ** 2 / (256 * m2 ** 2) + 2725 * d * n ** 2 / (3072 * m2)
            - 15 * d * m2 * PI * chil / (16 * n) - 35 * m2 ** 2 * PI * chil / (16 * n)
            + chil ** 2 * (375 * d ** 2 * m2 ** 2 + 1815 * d * m2 ** 3) / (256 * n) + 1645 * m2 ** 4 * chil ** 2 / (192 * n)])
    return out


def rotate(v, axis, angle):
    c, s = np.cos(angle), np.sin(angle)
    m = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]]) if axis == "z" else np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])
    return m @ v


def wave_p(p, f):
    """h+ and hx of IMRPhenomPv2."""
    m1, m2 = p["mass1"] * MSUN, p["mass2"] * MSUN
    s1, s2 = np.array(p["spin1"]), np.array(p["spin2"])
    M, q = m1 + m2, m1 / m2
    eta = m1 * m2 / (M * M)
    A1, A2 = 2 + 3 * m2 / (2 * m1), 2 + 3 * m1 / (2 * m2)
    perp = max(A1 * m1 ** 2 * np.hypot(s1[0], s1[1]), A2 * m2 ** 2 * np.hypot(s2[0], s2[1]))
    chip = perp / (A2 * m2 ** 2 if m2 > m1 else A1 * m1 ** 2)
    chil = (1 + q) / q * (m1 * s1[2] + m2 * s2[2]) / M
    fm1, fm2 = q / (1 + q), 1 / (1 + q)
    SP, SL = chip * fm1 ** 2, s1[2] * fm1 ** 2 + s2[2] * fm2 ** 2

    def orbital(v2):  # L / M^2 from (pi M f)^(2/3)
        return eta * (1 + (1.5 + eta / 6) * v2 + (3.375 - 19 * eta / 8 - eta * eta / 24) * v2 * v2) / v2 ** 0.5

    J = m1 ** 2 * s1 + m2 ** 2 * s2
    J[2] += M * M * orbital((PI * M * p["f_ref"]) ** (2 / 3))
    th, ph = np.arccos(J[2] / np.linalg.norm(J)), np.arctan2(J[1], J[0])
    ci, si = np.cos(p["incl_angle"]), np.sin(p["incl_angle"])
    N = np.array([si * np.cos(PI / 2 - p["phiRef"]), si * np.sin(PI / 2 - p["phiRef"]), ci])

    def to_j(v):
        return rotate(rotate(v, "z", -ph), "y", -th)

    n1 = to_j(N)
    kappa = -np.arctan2(n1[1], n1[0])
    n1 = rotate(n1, "z", kappa)
    l1 = rotate(to_j(np.array([0, 0, 1.0])), "z", kappa)
    alpha0, theta = np.arctan2(l1[1], l1[0]), np.arccos(n1[2])
    X = rotate(to_j(np.array([-ci * np.sin(p["phiRef"]), -ci * np.cos(p["phiRef"]), si])), "z", kappa)
    zeta = np.arctan2(X[0] * n1[2] - X[2] * n1[0], -X[1])
    d = PhenomD(p, spin_in_plane=chip)
    ca, ce = euler_coefficients(q, chil, chip)

    def angle(c, w):
        L = torch.log(w) if torch.is_tensor(w) else np.log(w)
        return c[0] / w + c[1] / w ** (2.0 / 3) + c[2] / w ** (1.0 / 3) + c[3] * L + c[4] * w ** (1.0 / 3)

    fr = d.xr / M
    nodes = np.linspace(0.8 * fr, 1.2 * fr, 10)
    val = np.array([-scalar(d.phase, M * v) for v in nodes])
    t_corr = spline_at(nodes, val, spline(nodes, val), fr, slope=True) / (2 * PI)
    x, w, wr = M * f, PI * M * f, PI * M * p["f_ref"]
    al = angle(ca, w) - angle(ca, wr) + alpha0
    ep = angle(ce, w) - angle(ce, wr)
    s = SP / (orbital(w ** (2.0 / 3)) + SL)
    cb = 1 / torch.sqrt(1 + s * s)
    c, sn = torch.sqrt((1 + cb) / 2), torch.sqrt((1 - cb) / 2)
    up = [sn ** 4, 2 * c * sn ** 3, 6 ** 0.5 * sn ** 2 * c ** 2, 2 * c ** 3 * sn, c ** 4]
    dn = [up[4], -up[3], up[2], -up[1], up[0]]
    ct, st = np.cos(theta), np.sin(theta)
    Y = [np.sqrt(5 / (64 * PI)) * (1 - ct) ** 2, np.sqrt(5 / (16 * PI)) * st * (1 - ct), np.sqrt(15 / (32 * PI)) * st ** 2,
         np.sqrt(5 / (16 * PI)) * st * (1 + ct), np.sqrt(5 / (64 * PI)) * (1 + ct) ** 2]
    hp = torch.zeros_like(f, dtype=torch.complex128)
    hc = torch.zeros_like(hp)
    for m in range(-2, 3):
        e = torch.polar(torch.ones_like(f), m * al)
        a, b = e.conj() * (dn[m + 2] * Y[m + 2]), e * (up[m + 2] * Y[m + 2])
        hp = hp + a + b
        hc = hc + 1j * (a - b)
    amp = torch.where(x > d.cut, 0.0, d.A0 * M ** (7 / 6) / (4 * np.sqrt(5 / (64 * PI))) * x ** (-7.0 / 6) * d.amplitude(x))
    phase = d.phase(x) + 2 * ep - turn(p["tc"], f - p["f_ref"]) + 2 * ph + 2 * PI * t_corr * f
    h = torch.polar(torch.ones_like(f), -phase) * amp
    hp, hc = hp * h, hc * h
    cz, sz = np.cos(2 * zeta), np.sin(2 * zeta)
    return cz * hp + sz * hc, cz * hc - sz * hp


def antenna(p, i):
    """F+, Fx of detector i and its arrival time after detector 0's."""
    t = tables()
    g, cd, sd = p["gmst"] - p["RA"], np.cos(p["DEC"]), np.sin(p["DEC"])
    cg, sg, cp, sp = np.cos(g), np.sin(g), np.cos(p["psi"]), np.sin(p["psi"])
    X = np.array([-cp * sg - sp * cg * sd, -cp * cg + sp * sg * sd, sp * cd])
    Y = np.array([sp * sg - cp * cg * sd, sp * cg + cp * sg * sd, cp * cd])
    D = t["tensor"][i] * t["geom"][i]
    e = np.array([cd * cg, -cd * sg, sd])
    return X @ D @ X - Y @ D @ Y, X @ D @ Y + Y @ D @ X, (t["loc"][0] - t["loc"][i]) @ e / C


def responses(p, model, f, dets):
    hp, hc = (wave_p if model == "P" else wave_d)(p, f)
    out = []
    for i in range(dets):
        fp, fc, dt = antenna(p, i)
        out.append((fp * hp + fc * hc) * torch.polar(torch.ones_like(f), -2 * PI * dt * f))
    return out


def simpson(f):
    n = f.size
    w = np.where(np.arange(n) % 2 == 1, 4.0, 2.0)
    w[0] = w[-1] = 1.0
    return w


def exact(case, seed):
    kind, model, dets = case["kind"], case["model"], case["dets"]
    if kind == "fisher":
        return None  # a difference quotient: its value is that of its own steps and rounding
    data, which = streams(case, seed)
    plist = parameters(case, seed + 1)
    dev = []
    for T, f, w, psd, dat in data:
        if w is not None:
            wt = 4.0 * w
        elif kind == "maximized":
            wt = 4.0 * (f[1] - f[0]) / 3.0 * simpson(f)
        else:
            wt = 4.0 * (f[f.size // 2] - f[f.size // 2 - 1]) / 3.0 * simpson(f)
        dev.append((T, torch.from_numpy(f).cuda(), torch.from_numpy(wt / psd).cuda(), torch.from_numpy(4.0 / psd).cuda(),
                    [torch.from_numpy(x).cuda() for x in dat]))
    out = []
    for p, g in zip(plist, which):
        T, f, wt, s4, dat = dev[g]
        if kind == "maximized":
            df = float(f[1] - f[0])
            p = dict(p, RA=0.0, DEC=0.0, psi=0.0, phiRef=1.0, tc=1.0, incl_angle=0.0, f_ref=20.0 if model == "P" else 10.0)
            hp, hc = (wave_p if model == "P" else wave_d)(p, f)
            ll = 0.0
            for d in dat:
                hh = (wt * hp.abs() ** 2).sum()
                gp = torch.fft.fft(s4 * d.conj() * hp)
                if model == "D":
                    ll = ll + 0.5 * (gp.abs() ** 2).max() * df * df / hh
                    continue
                cc = (wt * hc.abs() ** 2).sum()
                I = (wt * (hp * hc.conj()).real).sum() / torch.sqrt(hh * cc)
                rp, rc = gp * df / torch.sqrt(hh), torch.fft.fft(s4 * d.conj() * hc) * df / torch.sqrt(cc)
                a, b, gm = rp.abs() ** 2, rc.abs() ** 2, (rp * rc.conj()).real
                lam = (a + b - 2 * gm * I + torch.sqrt((a - b) ** 2 + 4 * (I * a - gm) * (I * b - gm))) / (1 - I * I)
                ll = ll + 0.25 * lam.max()
            out.append(ll)
        else:
            r = responses(dict(p, tc=T - p["tc"]), model, f, dets)
            out.append(sum((wt * ((d.conj() * x).real - 0.5 * x.abs() ** 2)).sum() for d, x in zip(dat, r)))
    ll = torch.stack(out).cpu().numpy()
    return ll if kind == "plain" else (ll, None)

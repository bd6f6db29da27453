// fisher_ff.h -- the Fisher moment form's per-bin differences and sums in two
// floats (two_float.h), host and device.
//
// The coefficients stay those of FisherSrc: the differences of the perturbed
// waveforms' FP64 coefficients, taken in FP64 and split into pairs.  At a bin
// where both waveforms of a pair are in the same regions, the difference is a
// short series in the per-bin powers, evaluated in two floats; the remaining
// bins (between the region boundaries of a pair, across a cut, pairs at
// eta = 1/4, steps too large for the series) are left to fisher_pair_q in FP64.
#pragma once

#include "fisher_math.h"
#include "phenom_acc.h"

namespace gwf {

// A position on the grid as an integer and a fraction: n - pos is exact to 2^-48.
struct FfPos {
  int n;
  ff frac;
};
struct FfPair {
  int n_cut, slow;      // last bin with both waveforms; 1: FP64 at every bin
  int a1, a2, a3, a4;   // amplitude: inspiral below a1, intermediate in [a2, a3), ringdown from a4
  int b1, b2, b3, b4;   // phase, the same way
  float div;
  ff hdiv;              // half the divisor
  ff qi[12], bi0, bi1;  // the differences of WaveDiff (phi_c within qi[5], pA, mA)
  ff pA, pB, pC, pD, mA, mB, mC, mD;
  ff ai[10], ei[5];
  // ringdown amplitude of the - waveform (K with its scale) and the parts of
  // ln(A+ / A-) / divisor: c0 + c1 x- + log1p(u) / div,
  // u / div = (e1 (x- + x+) + e2) / (x+^2 + gp)
  ff K, ex, gm, gp, c0, c1, e1, e2;
  FfPos rm, rp;
  // ringdown atan: y = (n - c) w, (y+ - y-) / div = f1 n + f2
  ff wm, wp, f1, f2, mE, dE;
  FfPos cm, cp;
};
struct FfSrc {
  int ok;  // 0: a coefficient that two floats cannot hold (FP64 sums then)
  int n_f1, n_f3, n_cut, n_cut_any, n_mid;
  ff ai[10], ei[5], K, ex, g;
  FfPos rd;
  FfPair q[kIntr];
};

GW_HD bool ff_set(ff &a, double v) {
  a = ff_split(v);
  return fabs(v) < 1e30;
}
GW_HD bool ff_set_pos(FfPos &p, double pos) {
  const bool ok = fabs(pos) < 16777216.0;
  const double f = ok ? floor(pos) : 0.0;
  p.n = (int)f;
  p.frac = ff_split(pos - f);
  return ok;
}
GW_HD ff ff_from(int n, const FfPos &p) {
  ff x = two_sum((float)(n - p.n), -p.frac.h);
  x.l -= p.frac.l;
  return x;
}

GW_HD int imin(int a, int b) { return a < b ? a : b; }
GW_HD int imax(int a, int b) { return a > b ? a : b; }

GW_HD bool ff_centre(const FisherSrc &F, FfSrc &S) {
  const WaveF64 &w = F.w0;
  bool ok = true;
  S.n_f1 = w.n_f1;
  S.n_f3 = w.n_f3;
  S.n_cut = w.n_cut;
  S.n_cut_any = F.n_cut_any;
  S.n_mid = w.n_mid;
  for (int j = 0; j < 10; j++) ok &= ff_set(S.ai[j], w.ai[j]);
  for (int j = 0; j < 5; j++) ok &= ff_set(S.ei[j], w.ei[j]);
  ok &= ff_set(S.K, w.mrK);
  ok &= ff_set(S.ex, w.mrExp);
  ok &= ff_set(S.g, w.mrG2);
  ok &= ff_set_pos(S.rd, w.nrd);
  return ok && w.n_mid > -16777216 && w.n_mid < 16777216;
}
// Of step threads part takes every step-th of the series, the first the rest.
GW_HD bool ff_pair(const FisherSrc &F, int q, FfPair &P, int part, int step) {
  const WaveF64 &p = F.wp[q], &m = F.wm[q];
  const WaveDiff &d = F.wd[q];
  const double inv = F.idiv[q], div = F.div[7 + q];
  bool ok = true;
  for (int j = part; j < 12; j += step) ok &= ff_set(P.qi[j], j == 5 ? d.qi[5] - d.phic : d.qi[j]);
  for (int j = part; j < 10; j += step) ok &= ff_set(P.ai[j], d.ai[j]);
  for (int j = part; j < 5; j += step) ok &= ff_set(P.ei[j], d.ei[j]);
  if (part) return ok;
  P.n_cut = imin(imin(p.n_cut, m.n_cut), F.w0.n_cut);
  P.slow = F.exact[q] || F.onesided[q];
  P.a1 = imin(p.n_f1, m.n_f1);
  P.a2 = imax(p.n_f1, m.n_f1);
  P.a3 = imin(p.n_f3, m.n_f3);
  P.a4 = imax(p.n_f3, m.n_f3);
  P.b1 = imin(p.n_f1p, m.n_f1p);
  P.b2 = imax(p.n_f1p, m.n_f1p);
  P.b3 = imin(p.n_f2p, m.n_f2p);
  P.b4 = imax(p.n_f2p, m.n_f2p);
  P.div = (float)div;
  ok &= ff_set(P.hdiv, 0.5 * div);
  ok &= ff_set(P.bi0, d.bi0);
  ok &= ff_set(P.bi1, d.bi1);
  ok &= ff_set(P.pA, d.pA - d.phic);
  ok &= ff_set(P.pB, d.pB);
  ok &= ff_set(P.pC, d.pC);
  ok &= ff_set(P.pD, -d.pD);
  ok &= ff_set(P.mA, d.mA - d.phic);
  ok &= ff_set(P.mB, d.mB);
  ok &= ff_set(P.mC, -d.mC);
  ok &= ff_set(P.mD, d.mD);
  ok &= ff_set(P.K, m.mrK * F.sm[q]);
  ok &= ff_set(P.ex, m.mrExp);
  ok &= ff_set(P.gm, m.mrG2);
  ok &= ff_set(P.gp, p.mrG2);
  ok &= ff_set(P.c0, (F.amp_lk[q] - p.mrExp * (m.nrd - p.nrd)) * inv);
  ok &= ff_set(P.c1, (m.mrExp - p.mrExp) * inv);
  ok &= ff_set(P.e1, (p.nrd - m.nrd) * inv);
  ok &= ff_set(P.e2, (m.mrG2 - p.mrG2) * inv);
  ok &= ff_set_pos(P.rm, m.nrd);
  ok &= ff_set_pos(P.rp, p.nrd);
  ok &= ff_set(P.wm, m.inv_nw);
  ok &= ff_set(P.wp, p.inv_nw);
  ok &= ff_set(P.f1, d.yw);
  ok &= ff_set(P.f2, d.yc);
  ok &= ff_set(P.mE, p.mE);
  ok &= ff_set(P.dE, (p.mE - m.mE) * inv);
  ok &= ff_set_pos(P.cm, m.nc);
  ok &= ff_set_pos(P.cp, p.nc);
  return ok;
}

// The per-bin powers.
struct FfBin {
  ff t, m76, i, ln, inv, t34;  // n^(1/3), n^(-7/6), n^(-1/3), ln n, 1/n, n^(3/4)
  float n;
};
GW_HD FfBin ff_bin(const AccTables &tb, int n) {
  const ff4 a = acc_ld(tb.pw + n), b = acc_ld(tb.pv + n), c = acc_ld(tb.ph + n);
  return FfBin{ff{a.ch, a.cl}, ff{a.sh, a.sl}, ff{b.ch, b.cl}, ff{b.sh, b.sl}, ff{c.ch, c.cl}, ff{c.sh, c.sl}, (float)n};
}
template <int N>
GW_HD ff ff_poly(const ff *c, ff x) {  // c[0] + c[1] x + .. + c[N-1] x^(N-1)
  ff a = c[N - 1];
#pragma unroll
  for (int j = N - 2; j >= 0; j--) a = ff_add(ff_mul(a, x), c[j]);
  return a;
}
template <int N>
GW_HD ff ff_polyf(const ff *c, float x) {
  ff a = c[N - 1];
#pragma unroll
  for (int j = N - 2; j >= 0; j--) a = ff_add(ff_mulf(a, x), c[j]);
  return a;
}

// The centre's amplitude / A_scale (0 beyond its cut).
GW_HD ff ff_amp0(const FfSrc &S, int n, const FfBin &b, const AccLut &lut) {
  if (n > S.n_cut) return ff{0.f, 0.f};
  ff a;
  if (n < S.n_f1) {
    a = ff_poly<10>(S.ai, b.t);
  } else if (n >= S.n_f3) {
    const ff x = ff_from(n, S.rd);
    const ff den = ff_norm(ff_add(ff_sqr(x), S.g));
    a = ff_div(ff_norm(ff_mul(ff_exp(ff_norm(ff_neg(ff_mul(S.ex, x))), lut.ex), S.K)), den);
  } else {
    a = ff_polyf<5>(S.ei, (float)(n - S.n_mid));
  }
  return ff_norm(ff_mul(ff_norm(a), b.m76));
}

// Pair q's difference at bin n relative to the centre's phase, per unit step,
// a0 the centre's amplitude; false where it is left to FP64.
GW_HD bool ff_pair_q(const FfPair &P, int n_mid, int n, const FfBin &b, const AccLut &lut, ff a0, ff &qr, ff &qi) {
  if (P.slow || n > P.n_cut || a0.h == 0.0f) return false;
  ff da, dp;
  if (n < P.b1) {
    ff lo = P.qi[0];
#pragma unroll
    for (int j = 1; j <= 5; j++) lo = ff_add(ff_mul(lo, b.i), P.qi[j]);
    const ff hi = ff_mul(ff_poly<6>(P.qi + 6, b.t), b.t);
    dp = ff_add(ff_add(lo, hi), ff_mul(b.ln, ff_norm(ff_add(P.bi0, ff_mul(P.bi1, b.t)))));
  } else if (n >= P.b2 && n < P.b3) {
    const ff i3 = ff_mul(ff_sqr(b.inv), b.inv);
    dp = ff_add(ff_add(ff_add(P.pA, ff_mulf(P.pB, b.n)), ff_mul(P.pC, b.ln)), ff_mul(P.pD, i3));
  } else if (n >= P.b4) {
    const ff ym = ff_norm(ff_mul(ff_from(n, P.cm), P.wm)), yp = ff_norm(ff_mul(ff_from(n, P.cp), P.wp));
    const ff den = ff_norm(ff_addf(ff_mul(yp, ym), 1.0f));
    const ff z = ff_div(ff_norm(ff_add(ff_mulf(P.f1, b.n), P.f2)), den);  // per unit step
    const float zz = z.h * P.div;
    if (!(fabsf(zz) < 1e-3f)) return false;
    const float z2 = zz * zz;
    const ff at = ff_add(z, ff_mulf(z, -z2 * ((1.0f / 3.0f) - z2 * 0.2f)));
    ff d;
    const int i = ff_atan(ym, lut.turn, d);
    const double step = 6.28318530717958647692 / kTurnTab;
    const ff am = ff_norm(ff_add(ff_mulf(ff{(float)step, (float)(step - (double)(float)step)}, (float)i), d));
    dp = ff_add(ff_add(P.mA, ff_mulf(P.mB, b.n)), ff_add(ff_mul(P.mC, b.inv), ff_mul(P.mD, b.t34)));
    dp = ff_add(dp, ff_add(ff_mul(P.mE, ff_norm(at)), ff_mul(P.dE, am)));
  } else {
    return false;
  }
  if (n < P.a1) {
    da = ff_mul(ff_norm(ff_poly<10>(P.ai, b.t)), b.m76);
  } else if (n >= P.a2 && n < P.a3) {
    da = ff_mul(ff_norm(ff_polyf<5>(P.ei, (float)(n - n_mid))), b.m76);
  } else if (n >= P.a4) {
    const ff xm = ff_from(n, P.rm), xp = ff_from(n, P.rp);
    const ff dm = ff_norm(ff_add(ff_sqr(xm), P.gm)), dq = ff_norm(ff_add(ff_sqr(xp), P.gp));
    const ff u = ff_div(ff_norm(ff_add(ff_mul(P.e1, ff_norm(ff_add(xm, xp))), P.e2)), dq);
    const float uu = u.h * P.div;
    ff L = ff_add(ff_add(P.c0, ff_mul(P.c1, xm)), ff_add(u, ff_mulf(u, -uu * (0.5f - uu * (1.0f / 3.0f)))));
    L = ff_norm(L);
    const float LL = L.h * P.div;
    if (!(fabsf(uu) < 1e-4f && fabsf(LL) < 1e-4f)) return false;
    L = ff_add(L, ff_mulf(L, LL * (0.5f + LL * (1.0f / 6.0f))));
    const ff e = ff_norm(ff_mul(ff_exp(ff_norm(ff_neg(ff_mul(P.ex, xm))), lut.ex), P.K));
    da = ff_mul(ff_norm(ff_mul(ff_div(e, dm), b.m76)), ff_norm(L));
  } else {
    return false;
  }
  // cos h and sin h / h of half the phase step: h stays below 1e-2
  dp = ff_norm(dp);
  const ff h = ff_norm(ff_mul(dp, P.hdiv));
  if (!(fabsf(h.h) < 0.03f)) return false;
  const ff h2 = ff_sqr(h);
  const float h4 = h2.h * h2.h;
  const ff ec{0.5f * h2.h, f_fma(h4, -1.0f / 24.0f, 0.5f * h2.l)};  // 1 - cos h
  const double six = 1.0 / 6.0;
  ff es = ff_mul(h2, ff{(float)six, (float)(six - (double)(float)six)});  // 1 - sin h / h
  es.l = f_fma(h4, -1.0f / 120.0f, es.l);
  da = ff_norm(da);
  qr = ff_norm(ff_sub(da, ff_mul(da, ec)));
  const ff v = ff_norm(ff_mul(a0, dp));
  qi = ff_norm(ff_sub(ff_mul(v, es), v));
  return true;
}

// The moment sums, with the bin number for the frequency.
GW_HD void ff_accumulate(ff w, ff a0, float n, const ff *qr, const ff *qi, ff *A) {
  const ff wa = ff_norm(ff_mul(w, a0));
  const ff m0 = ff_norm(ff_mul(wa, a0)), m1 = ff_norm(ff_mulf(m0, n));
  ff_acc(A[0], m0);
  ff_acc(A[1], m1);
  ff_acc(A[2], ff_mulf(m1, n));
  int o = 3;
#pragma unroll
  for (int i = 0; i < kIntr; i++) {
    const ff wr = ff_norm(ff_mul(w, qr[i])), wi = ff_norm(ff_mul(w, qi[i]));
#pragma unroll
    for (int j = i; j < kIntr; j++) ff_acc(A[o++], ff_add(ff_mul(wr, qr[j]), ff_mul(wi, qi[j])));
    const ff sr = ff_norm(ff_mul(wr, a0)), si = ff_norm(ff_mul(wi, a0));
    ff_acc(A[13 + 4 * i + 0], sr);
    ff_acc(A[13 + 4 * i + 1], si);
    ff_acc(A[13 + 4 * i + 2], ff_mulf(sr, n));
    ff_acc(A[13 + 4 * i + 3], ff_mulf(si, n));
  }
}

}  // namespace gwf

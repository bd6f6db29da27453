// phenom_acc.h -- the FP64 form's bins in two-float arithmetic (host and device).
//
// The same quantity as phenom_mixed.h, on grids of n dfq (acc_on_line) or of
// nodes, to FP64 accuracy: what is linear in n in the phase is exact
// 64-bit fixed-point turns, the inspiral and intermediate phase series (up to
// 1e4 rad) stay FP64, and everything of order one -- amplitude, ringdown phase,
// sine and cosine, projection, data products, sums -- is carried on pairs of
// FP32 numbers (two_float.h, 48 bits).  GB300 issues 64 FP32 instructions in
// the time of an FP64 one, and FP64 bins spend ~290 FP64 instructions each
// (18,900 cycles per warp); the two-float IMRPhenomD bin is ~550 FP32
// instructions.  The rounding of a bin, ~1e-14, stays below that of its FP64
// phase, ~1e-12 rad.
#pragma once

#include <cstring>
#include <type_traits>

#include "phenom_mixed.h"
#include "two_float.h"

namespace gwt {

// Tables by n for the two-float bins, and the FP64 powers the phase series take.
struct AccTables {
  const ff4 *pw;       // n^(1/3), n^(-7/6)
  const ff4 *ph;       // 1/n, n^(3/4)
  const ff4 *pv;       // n^(-1/3), ln n
  const double *t13, *tm53, *tln, *t34;  // n^(1/3), n^(-5/3), ln n, n^(3/4)
  int nmax;            // valid for 1 <= n <= nmax
};

// A grid of any other spacing (quadrature nodes; acc_on_line): bins at x = f / df, df the
// power of two that puts the highest frequency in [2^19, 2^20); the weights and
// data products as on uniform grids, the tables by the bin's index.
constexpr int kNodeBits = 42;
struct AccNodes {
  const ff4 *wd;
  const ff *wf;
  AccTables tb;
  const int64_t *X;  // x 2^kNodeBits
  const ff *x;
};

// Sine/cosine and exponential tables (shared memory in the kernels).
struct AccLut {
  ff4 turn[kTurnTab];
  ff ex[kExpTab];
};

// Largest bin count whose indices are exact in FP32.
constexpr int kAccMaxN = 1 << 24;
// Largest phase term carried in two floats, in turns: its rounding, ~4e-15 of it,
// must stay below the FP64 series' own.
constexpr double kAccMaxTurns = 12.0;

// Constants of one request: the mixed form's (regions, FP64 phase
// coefficients, hi/lo amplitude coefficients, final factors) and what the
// two-float bins need beside them.
struct AccReq {
  MixedReq m;
  uint64_t L0[kMaxDet], L1[kMaxDet];  // linear phase of each detector, turns 2^64: L0 + L1 n
  uint64_t B0, B1;                    // the same without a detector's delay and projection phase
  uint64_t pR0, pR1;                  // intermediate phase: its constant and linear terms
  uint64_t mR0, mR1;                  // ringdown phase: the same
  uint64_t mEq;                       // ringdown: mE / kTurnTab (mE atan at the table angles)
  ff rdfrac, ncfrac, inv_nw;          // n_rd, n_c and the atan width to two floats
  ff cC, cD, cE;                      // ringdown terms in turns: cC / n + cD n^(3/4) + cE (atan remainder)
  // Pv2: alpha and 2 epsilon in turns, ((a0 i + a1) i + a2) i + a3 t + a4 ln n + const (i = n^(-1/3));
  ff al[5], ep[5];
  uint64_t alQ, epQ;
  ff us[4];                           // 1/s = us0 i + us1 t + us2 n + us3 (the Wigner angle)
  ff y2p, y1p, y0p, y2m, y1m;         // harmonics: sums and differences of Y_m and Y_-m
  ff c2z, s2z;                        // polarisation rotation
  float tc;                           // model's t_c, for the rounding of a bin's frequency (acc_dev_turns)
  float bad;                          // NaN when a linear phase is (turns cannot hold it), else 0; joins the result
  // On nodes (acc_node_coeffs): slopes of the linear phases in turns per bin
  // 2^(node_shift + 64 - kNodeBits), region boundaries as the bits of the
  // frequencies (f positive: ordered as integers), n_rd and n_c whole
  int64_t nS[kMaxDet], nP, nM;
  int64_t f1, f1p, f3, f2p, fcut;
  ff nrd, nc;
  int node_shift;
  int fp64_phase;                     // 1: terms too large for two floats; every bin takes the FP64 series
};

// Turns to 2^64 per turn.  The nearest whole turn is taken off, which is exact
// and leaves a small count (a phase step per bin) all its digits: the step is
// multiplied by n.
GW_HD uint64_t acc_turns(double t) {
  t -= rint(t);
  return (uint64_t)gw_llrint(t * 9223372036854775808.0) << 1;
}
// a b turns, the product's rounding error included.
GW_HD uint64_t acc_turns_prod(double a, double b) {
  const double p = a * b;
  return acc_turns(p) + acc_turns(fma(a, b, -p));
}
GW_HD uint64_t radians_q64(double ph) { return acc_turns(ph * (1.0 / (2.0 * 3.14159265358979323846))); }

// ---- prologue parts, after the mixed form's of the same request ----
// Detector phases (as mixed_det_phase): t_c enters as turns, t_c f, so that the
// whole turns of a long segment leave no rounding behind.  Detectors d0, d0 + step, ...
GW_HD void acc_det_phase(const Request &r, double df, AccReq &x, int d0 = 0, int step = 1) {
  const ModelD &m = r.m;
  const bool pv2 = r.approximant == kPhenomPv2;
  const double inv2pi = 1.0 / (2.0 * kPi);
  const uint64_t q0 = acc_turns_prod(m.s.tc, m.fref) + acc_turns((m.tcs * m.fref - m.phic) * inv2pi);
  const double c1 = pv2 ? r.p.t_corr * df : -m.tcs * df * inv2pi;
  const uint64_t q1 = acc_turns(c1) - acc_turns_prod(m.s.tc, df);
  x.tc = (float)m.s.tc;
  x.bad = (float)(0.0 * (m.s.tc * m.fref + m.tcs * m.fref - m.phic + c1));
  x.B0 = q0;
  x.B1 = q1;
  for (int d = d0; d < r.ndet && d < kMaxDet; d += step) {
    double Gre, Gim;
    mixed_det_G(r, d, Gre, Gim);
    x.L0[d] = q0;
    x.L1[d] = q1 - acc_turns(r.det[d].tau * df * inv2pi);
    if (!pv2) x.L0[d] -= acc_turns(atan2(Gim, Gre) * inv2pi);
  }
}
GW_HD void acc_phase_coeffs(const Request &r, double df, AccReq &x) {
  const double inv2pi = 1.0 / (2.0 * kPi);
  const MixedReq &m = x.m;
  x.pR0 = acc_turns(m.pA * inv2pi);
  x.pR1 = acc_turns(m.pB * inv2pi);
  x.mR0 = acc_turns(m.mA * inv2pi);
  x.mR1 = acc_turns(m.mB * inv2pi);
  x.mEq = acc_turns(m.mE * inv2pi * (2.0 * kPi / kTurnTab));
  x.cC = ff_split(-m.mC * inv2pi);
  x.cD = ff_split(m.mD * inv2pi);
  x.cE = ff_split(m.mE * inv2pi);
  const Source &s = r.m.s;
  const double nc = r.m.l.alpha[5] * s.fRD / df;
  x.ncfrac = ff_split(nc - floor(nc));
  x.inv_nw = ff_split(df / s.fdamp);
}
GW_HD void acc_amp_coeffs(const Request &r, double df, AccReq &x) {
  const double nrd = r.m.s.fRD / df;
  x.rdfrac = ff_split(nrd - floor(nrd));
}
GW_HD int64_t acc_bits(double v) {
  int64_t b;
  memcpy(&b, &v, 8);
  return b;
}
// What nodes need beside the above (df: their scale), the linear phases first:
// a slope of at most 2^62 in size against x 2^kNodeBits, a 128-bit product.
GW_HDNI void acc_node_coeffs(const Request &r, double df, AccReq &x) {
  const ModelD &m = r.m;
  const double inv2pi = 1.0 / (2.0 * kPi);
  const double c1 = r.approximant == kPhenomPv2 ? r.p.t_corr * df : -m.tcs * df * inv2pi, tc = m.s.tc * df;
  double tau[kMaxDet], big = 0.0;
  for (int d = 0; d < r.ndet && d < kMaxDet; d++) {
    tau[d] = r.det[d].tau * df * inv2pi;
    big = fmax(big, fabs(tau[d]));
  }
  const double pB = x.m.pB * inv2pi, mB = x.m.mB * inv2pi;
  big += fabs(c1) + fabs(tc) + fabs(pB) + fabs(mB);
  int a = big > 0.0 && big < 1e300 ? 61 - ilogb(big) : 85;
  a = a > 85 ? 85 : a < 23 ? 23 : a;
  // beyond 2^38 turns per bin no digit of a bin's phase is left
  const double sc = big < 274877906944.0 ? ldexp(1.0, a) : 0.0;
  for (int d = 0; d < r.ndet && d < kMaxDet; d++)
    x.nS[d] = gw_llrint(c1 * sc) - gw_llrint(tc * sc) - gw_llrint(tau[d] * sc);
  x.nP = gw_llrint(pB * sc);
  x.nM = gw_llrint(mB * sc);
  x.node_shift = a + kNodeBits - 64;
  x.f1 = acc_bits(m.s.f1);
  x.f1p = acc_bits(m.s.f1_phase);
  x.f3 = acc_bits(m.s.f3);
  x.f2p = acc_bits(m.s.f2_phase);
  x.fcut = acc_bits(m.fcut);
  x.nrd = ff_split(m.s.fRD / df);
  x.nc = ff_split(m.l.alpha[5] * m.s.fRD / df);
}
// Pv2, after mixed_pv2_coeffs and mixed_phase_coeffs: epsilon joins the
// inspiral phase series (the same powers of n), the rest in turns.
GW_HD void acc_pv2_coeffs(const Request &r, double df, AccReq &x) {
  MixedReq &m = x.m;
  const double inv2pi = 1.0 / (2.0 * kPi);
  m.qi[2] += 2.0 * m.ee[0];
  m.qi[3] += 2.0 * m.ee[1];
  m.qi[4] += 2.0 * m.ee[2];
  m.qi[5] += 2.0 * m.ee[3];
  m.qi[6] += 2.0 * m.ee[4];
  m.bi0 += 2.0 * m.ee[5];
  for (int j = 0; j < 3; j++) {
    x.al[j] = ff_split(m.ea[j] * inv2pi);
    x.ep[j] = ff_split(2.0 * m.ee[j] * inv2pi);
  }
  x.al[3] = ff_split(m.ea[4] * inv2pi);
  x.al[4] = ff_split(m.ea[5] * inv2pi);
  x.ep[3] = ff_split(2.0 * m.ee[4] * inv2pi);
  x.ep[4] = ff_split(2.0 * m.ee[5] * inv2pi);
  x.alQ = acc_turns(m.ea[3] * inv2pi);
  x.epQ = acc_turns(2.0 * m.ee[3] * inv2pi);
  const Source &s = r.m.s;
  const double eta = s.eta, l1 = 1.5 + eta / 6.0, l2 = 3.375 - (19.0 * eta) / 8. - eta * eta / 24.0;
  // x = cw^2 t^2; only |1/s| enters.  No in-plane spin (SP = 0): 1/s stays finite and the angle is below 1e-20
  const double cw = cbrt(kPi * s.M * df), sp = fabs(s.SP), iSP = 1.0 / (sp < 1e-25 ? 1e-25 : sp);
  x.us[0] = ff_split(eta * iSP / cw);
  x.us[1] = ff_split(eta * l1 * iSP * cw);
  x.us[2] = ff_split(eta * l2 * iSP * (cw * cw * cw));
  x.us[3] = ff_split(s.SL * iSP);
  const double *Y = r.p.Y;  // m = -2..2
  x.y2p = ff_split(Y[4] + Y[0]);
  x.y1p = ff_split(Y[3] - Y[1]);
  x.y0p = ff_split(2.0 * kSqrt6 * 0.25 * Y[2]);
  x.y2m = ff_split(Y[0] - Y[4]);
  x.y1m = ff_split(-Y[1] - Y[3]);
  x.c2z = ff_split(r.p.c2z);
  x.s2z = ff_split(r.p.s2z);
}
// Whether the terms that the bins carry in two floats are small enough: their
// rounding, ~4e-15 of the largest, must stay below the FP64 series' own.
GW_HD void acc_range(const Request &r, AccReq &x) {
  const MixedReq &m = x.m;
  const double na = m.n_f1p > 1 ? m.n_f1p : 1, nb = m.n_cut > na ? m.n_cut : na;
  const double q = sqrt(nb);
  double v = fabs(ff_value(x.cC)) / na + fabs(ff_value(x.cD)) * (q * sqrt(q)) + fabs(ff_value(x.cE));
  if (r.approximant == kPhenomPv2) {
    const double i = 1.0 / cbrt(na), t = cbrt(nb), l = log(nb);
    double va = 0.0, ve = 0.0;
    for (int j = 0; j < 3; j++) {
      va = (va + fabs(ff_value(x.al[j]))) * i;
      ve = (ve + fabs(ff_value(x.ep[j]))) * i;
    }
    va += fabs(ff_value(x.al[3])) * t + fabs(ff_value(x.al[4])) * l;
    ve += fabs(ff_value(x.ep[3])) * t + fabs(ff_value(x.ep[4])) * l;
    v = fmax(v, fmax(va, ve));
  }
  x.fp64_phase = v < kAccMaxTurns ? 0 : 1;  // also for NaN
}
// The whole request after request_prologue (one thread; the check of phenom_fast.h's).
GW_HDNI int acc_prologue(const Request &r, double df, AccReq &x, const double *dscale, const double *wscale) {
  mixed_prologue(r, df, x.m, dscale, wscale);
  acc_det_phase(r, df, x);
  acc_phase_coeffs(r, df, x);
  acc_amp_coeffs(r, df, x);
  if (r.approximant == kPhenomPv2) acc_pv2_coeffs(r, df, x);
  acc_range(r, x);
  return x.m.status;
}

// ---- bins ----
GW_HD ff acc_pair(const float *h, const float *l, int j) { return ff{h[j], l[j]}; }
GW_HD double acc_ld(const double *p) {
#if defined(__CUDA_ARCH__)
  return __ldg(p);
#else
  return *p;
#endif
}
GW_HD ff4 acc_ld(const ff4 *p) {
#if defined(__CUDA_ARCH__)
  const float4 v = __ldg((const float4 *)p);
  return ff4{v.x, v.y, v.z, v.w};
#else
  return *p;
#endif
}
// A bin of a uniform grid (qd: its acc_dev_turns) and a node (f's bits, x 2^kNodeBits,
// x; sl: the slope of its phase region).  The functions below take either.
struct AccBin {
  int n;
  uint64_t qd;
};
struct AccNode {
  int k;
  int64_t f, X;
  ff x;
  int64_t sl;
};
GW_HD int acc_at(const AccBin &b) { return b.n; }
GW_HD int acc_at(const AccNode &b) { return b.k; }
GW_HD bool acc_ins_amp(const AccReq &x, const AccBin &b) { return b.n < x.m.n_f1; }
GW_HD bool acc_ins_amp(const AccReq &x, const AccNode &b) { return b.f < x.f1; }
GW_HD bool acc_ring_amp(const AccReq &x, const AccBin &b) { return b.n >= x.m.n_f3; }
GW_HD bool acc_ring_amp(const AccReq &x, const AccNode &b) { return b.f > x.f3; }
GW_HD bool acc_ins_phase(const AccReq &x, const AccBin &b) { return b.n < x.m.n_f1p; }
GW_HD bool acc_ins_phase(const AccReq &x, const AccNode &b) { return b.f < x.f1p; }
GW_HD bool acc_ring_phase(const AccReq &x, const AccBin &b) { return b.n >= x.m.n_f2p; }
GW_HD bool acc_ring_phase(const AccReq &x, const AccNode &b) { return b.f > x.f2p; }
// The bin's distance from a position, n0 + frac or whole.
GW_HD ff acc_from(const AccBin &b, int n0, ff frac, ff) {
  ff xx = two_sum((float)(b.n - n0), -frac.h);
  xx.l = f_sub(xx.l, frac.l);
  return xx;
}
GW_HD ff acc_from(const AccNode &b, int, ff, ff whole) { return ff_norm(ff_sub(b.x, whole)); }
GW_HD ff acc_times(ff a, const AccBin &b, int n0) { return ff_mulf(a, (float)(b.n - n0)); }
GW_HD ff acc_times(ff a, const AccNode &b, int n0) { return ff_mul(a, n0 ? ff_norm(ff_addf(b.x, -(float)n0)) : b.x); }
// S X 2^-s modulo one turn.
GW_HD uint64_t acc_node_turns(int64_t S, int64_t X, int s) {
#if defined(__CUDA_ARCH__)
  const uint64_t hi = (uint64_t)__mul64hi(S, X), lo = (uint64_t)S * (uint64_t)X;
#else
  const __int128 p = (__int128)S * X;
  const uint64_t hi = (uint64_t)(p >> 64), lo = (uint64_t)p;
#endif
  return (hi << (64 - s)) | (lo >> s);  // 1 <= s <= 63
}
// Detector d's linear phase (a node's with its region's slope).
GW_HD uint64_t acc_linear(const AccReq &x, const AccBin &b, int d) { return x.L0[d] + x.L1[d] * (uint64_t)b.n; }
GW_HD uint64_t acc_linear(const AccReq &x, const AccNode &b, int d) {
  return x.L0[d] + acc_node_turns(x.nS[d] + b.sl, b.X, x.node_shift);
}
GW_HD uint64_t acc_region_slope(const AccBin &b, uint64_t per_bin, int64_t) { return per_bin * (uint64_t)b.n; }
GW_HD uint64_t acc_region_slope(AccNode &b, uint64_t, int64_t sl) {
  b.sl = sl;
  return 0;
}
GW_HD uint64_t acc_offset(const AccBin &b) { return b.qd; }
GW_HD uint64_t acc_offset(const AccNode &) { return 0; }

// The FP64 phase of a bin in turns 2^64 without the linear terms (Pv2: with
// 2 epsilon), and alpha.
template <bool PV2, class B>
GW_HD uint64_t acc_phase64(const AccReq &x, B &b, const AccTables &tb, const AccLut &lut, uint64_t &al) {
  const MixedReq &m = x.m;
  const int n = acc_at(b);
  const double t = acc_ld(tb.t13 + n), r = acc_ld(tb.tm53 + n), lnn = acc_ld(tb.tln + n);
  double nd, eps = 0.0;
  if constexpr (std::is_same<B, AccBin>::value) {
    nd = (double)n;
    if (PV2) al = radians_q64(mixed_pv2_alpha(m, n, t, r, lnn));
    if (acc_ins_phase(x, b)) return radians_q64(mixed_phase_d(m, n, t, r, lnn, 0.0));
    if (PV2) eps = mixed_pv2_eps(m, n, t, r, lnn);
  } else {
    nd = (double)b.X * (1.0 / 4398046511104.0);
    b.sl = 0;
    if (PV2) {
      const double *a = m.ea, *e = m.ee;
      al = radians_q64(r * (a[0] * t * t + a[1] * nd + a[2] * nd * t) + a[3] + a[4] * t + a[5] * lnn);
      eps = r * (e[0] * t * t + e[1] * nd + e[2] * nd * t) + e[3] + e[4] * t + e[5] * lnn;
    }
    if (acc_ins_phase(x, b)) {
      double p = m.qi[11];
      for (int j = 10; j >= 0; j--) p = p * t + m.qi[j];
      return radians_q64(r * p + lnn * (m.bi0 + m.bi1 * t));
    }
  }
  double ph;
  uint64_t q = 0;
  if (acc_ring_phase(x, b)) {
    // the atan by its two-float form, |mE| ~ 1
    ff d;
    const int i = ff_atan(ff_norm(ff_mul(acc_from(b, m.n_c, x.ncfrac, x.nc), x.inv_nw)), lut.turn, d);
    ph = m.mA + m.mB * nd - m.mC * (r * t * t) + m.mD * acc_ld(tb.t34 + n) + m.mE * ff_value(d);
    q = x.mEq * (uint64_t)(int64_t)i;
  } else {
    ph = m.pA + m.pB * nd + m.pC * lnn - m.pD * (r * r * t);
  }
  if (PV2) ph += 2.0 * eps;
  return q + radians_q64(ph);
}
template <bool PV2, class B>
GW_HD uint64_t acc_phase(const AccReq &x, B &b, const AccTables &tb, const AccLut &lut, ff t, uint64_t &al) {
  const MixedReq &m = x.m;
  const int n = acc_at(b);
  if (acc_ins_phase(x, b) || x.fp64_phase) return acc_phase64<PV2>(x, b, tb, lut, al);
  uint64_t q;
  if (acc_ring_phase(x, b)) {
    const ff4 w = acc_ld(tb.ph + n);
    ff d;
    const int i = ff_atan(ff_norm(ff_mul(acc_from(b, m.n_c, x.ncfrac, x.nc), x.inv_nw)), lut.turn, d);
    ff v = ff_add(ff_mul(x.cD, ff{w.sh, w.sl}), ff_mul(x.cC, ff{w.ch, w.cl}));
    v = ff_add(v, ff_mul(x.cE, d));
    q = x.mR0 + acc_region_slope(b, x.mR1, x.nM) + x.mEq * (uint64_t)(int64_t)i + ff_turns_q64(ff_norm(v));
  } else {
    const double r = acc_ld(tb.tm53 + n);
    q = x.pR0 + acc_region_slope(b, x.pR1, x.nP) +
        radians_q64(m.pC * acc_ld(tb.tln + n) - m.pD * (r * r * acc_ld(tb.t13 + n)));
  }
  if (PV2) {
    const ff4 w = acc_ld(tb.pv + n);
    const ff i{w.ch, w.cl}, ln{w.sh, w.sl};
    ff a = ff_mul(ff_add(ff_mul(ff_add(ff_mul(x.al[0], i), x.al[1]), i), x.al[2]), i);
    a = ff_add(ff_add(a, ff_mul(x.al[3], t)), ff_mul(x.al[4], ln));
    al = x.alQ + ff_turns_q64(ff_norm(a));
    ff e = ff_mul(ff_add(ff_mul(ff_add(ff_mul(x.ep[0], i), x.ep[1]), i), x.ep[2]), i);
    e = ff_add(ff_add(e, ff_mul(x.ep[3], t)), ff_mul(x.ep[4], ln));
    q += x.epQ + ff_turns_q64(ff_norm(e));
  }
  return q;
}
// Amplitude / A_scale of a bin (below the cut): mixed_amp's formulas.
template <class B>
GW_HD ff acc_amp(const AccReq &x, const B &b, ff t, ff m76, const AccLut &lut) {
  const MixedReq &m = x.m;
  ff a;
  if (acc_ins_amp(x, b)) {
    a = acc_pair(m.ai, m.ai_lo, 9);
#pragma unroll
    for (int j = 8; j >= 0; j--) a = ff_add(ff_mul(a, t), acc_pair(m.ai, m.ai_lo, j));
  } else if (acc_ring_amp(x, b)) {
    const ff xx = acc_from(b, m.n_rd, x.rdfrac, x.nrd);
    const ff z = ff_norm(ff_neg(ff_mul(ff{m.mrExp, m.mrExp_lo}, xx)));
    const ff den = ff_norm(ff_add(ff_sqr(xx), ff{m.mrG2, m.mrG2_lo}));
    a = ff_div(ff_norm(ff_mul(ff_exp(z, lut.ex), ff{m.mrK, m.mrK_lo})), den);
  } else {
    a = acc_pair(m.ei, m.ei_lo, 4);
#pragma unroll
    for (int j = 3; j >= 0; j--) a = ff_add(acc_times(a, b, m.n_mid), acc_pair(m.ei, m.ei_lo, j));
  }
  return ff_norm(ff_mul(ff_norm(a), m76));
}

// The bins' rule: a uniform grid's bins are taken at n dfq, dfq = f_last / n_last,
// where every frequency is n dfq to its own rounding, four units in its last
// place (k (1 / T) and f0 + k df round to two).  What a bin's distance leaves
// out is then below FP64's own rounding of the phase: 2 pi tau(f) 2^-50 f for the
// series, whose time to coalescence tau falls from about T at the lowest
// frequencies as f^(-8/3), and as little for an arrival time; t_c is as large
// at every frequency and joins by acc_dev_turns.  Any other grid, 1e-9 of a bin
// off or drifting by as much, takes the node arrays, which hold f itself.
GW_HD double acc_spacing(double f_last, int n_last) { return f_last / n_last; }
GW_HD double acc_off_line(double f, int n, double dfq) { return fma(-(double)n, dfq, f); }
GW_HD bool acc_on_line(double f, double off) { return fabs(off) <= 0x1p-50 * f; }
// Phase of t_c at such a bin, whose frequency lies dev Hz off n dfq: |tc dev| is
// 1e-11 turn on a segment of 32 s, 2e-3 for a t_c counted in GPS seconds.  In two
// 32-bit conversions (2^-23 turn, the rest in 2^-55): one of 64 bits takes 1 % of
// the FP64 IMRPhenomD batch.
GW_HD uint64_t acc_dev_turns(const AccReq &x, float dev) {
  const float t = f_mul(-x.tc, dev);
  const int hi = f_to_int(f_mul(t, 8388608.0f));
  const int lo = f_to_int(f_mul(f_fma((float)hi, -1.0f / 8388608.0f, t), 36028797018963968.0f));
  return ((uint64_t)(int64_t)hi << 41) + ((uint64_t)(int64_t)lo << 9);
}

// IMRPhenomD bin: acc[2 d] weighted |h|^2 (detector 0 only when the detectors
// share their weights), acc[2 d + 1] Re(d* h e^{i phi_d}).  wd: the detector
// streams at this bin, W d (re, im); w: W.
template <int NDET, class B>
GW_HD void acc_bin_d(const AccReq &x, B b, const AccTables &tb, const AccLut &lut, const ff4 *wd, const ff *w,
                     bool wshared, ff *acc) {
  const ff4 p = acc_ld(tb.pw + acc_at(b));
  const ff t{p.ch, p.cl};
  const ff a = acc_amp(x, b, t, ff{p.sh, p.sl}, lut);
  uint64_t al;
  const uint64_t ph = acc_offset(b) + acc_phase<false>(x, b, tb, lut, t, al);
  const ff aa = ff_norm(ff_sqr(a));
#pragma unroll
  for (int d = 0; d < NDET; d++) {
    ff c, s;
    ff_turns_sincos(ph + acc_linear(x, b, d), lut.turn, c, s);
    if (d == 0 || !wshared) ff_acc(acc[2 * d], ff_mul(w[d], aa));
    const ff v = ff_sub(ff_mul(ff{wd[d].ch, wd[d].cl}, c), ff_mul(ff{wd[d].sh, wd[d].sl}, s));
    ff_acc(acc[2 * d + 1], ff_mul(a, v));
  }
}
// The IMRPhenomPv2 twist-up factors of bin n.  With cb, sb the cosine and sine of beta,
//   h+ = p2 (1 + cb^2)/2 cos 2a + p1 sb cb cos a + p0 sb^2 + i (p2 cb sin 2a + p1 sb sin a)
//   hx = i (m2 cb cos 2a + m1 sb cos a) - (m2 (1 + cb^2)/2 sin 2a + m1 sb cb sin a)
// (the half-angle products of IMRPhenomP.cpp:665-715 collected by e^{i k alpha}).
template <class B>
GW_HD void acc_twist(const AccReq &x, const B &b, const AccTables &tb, const AccLut &lut, ff t, uint64_t al, ff &hpr,
                     ff &hpi, ff &hcr, ff &hci) {
  const ff4 iw = acc_ld(tb.pv + acc_at(b));
  ff u = ff_add(ff_mul(x.us[0], ff{iw.ch, iw.cl}), ff_mul(x.us[1], t));
  u = ff_norm(ff_add(ff_add(u, acc_times(x.us[2], b, 0)), x.us[3]));
  ff cb, sb;
  if (fabsf(u.h) < 1e6f) {
    sb = ff_rsqrt(ff_norm(ff_addf(ff_sqr(u), 1.0f)));
    cb = ff_norm(ff_mul(u.h < 0.0f ? ff_neg(u) : u, sb));
  } else {
    // beta below 1e-6: as the reference's half angles of cos beta = 1 / sqrt(1 + s^2)
    // make it, whose distance from 1 is a whole number of 2^-52 there (1 + s^2
    // rounds to 1 + j 2^-52, its root down to half of that); NaN stays NaN
    const ff s = ff_div(ff{67108864.0f, 0.0f}, u), s2 = ff_norm(ff_sqr(s));  // 2^26 / u
    int j = f_to_int(s2.h);
    const float d = f_add(f_sub(s2.h, (float)j), s2.l);
    j += d > 0.5f ? 1 : d < -0.5f ? -1 : 0;
    const float r = (float)(j >> 1);
    sb = ff{sqrtf(r) * 2.1073424255447017e-08f, 0.0f};  // 2 sqrt(r 2^-53)
    cb = ff{u.h == u.h ? 1.0f : u.h, r * -2.2204460492503131e-16f};
  }
  ff ca, sa;
  ff_turns_sincos(al, lut.turn, ca, sa);
  const ff s2 = ff_norm(ff_mul(ff{2.0f * sa.h, 2.0f * sa.l}, ca));
  const ff ss = ff_sqr(sa);
  const ff c2 = ff_norm(ff_addf(ff{-2.0f * ss.h, -2.0f * ss.l}, 1.0f));
  const ff cc = ff_norm(ff_sqr(cb));
  const ff hc2{0.5f * cc.h, 0.5f * cc.l};
  const ff uu = ff_norm(ff_addf(hc2, 0.5f)), sc = ff_norm(ff_mul(sb, cb)), sq = ff_norm(ff_sqr(sb));
  hpr = ff_norm(ff_add(ff_add(ff_mul(ff_norm(ff_mul(x.y2p, uu)), c2), ff_mul(ff_norm(ff_mul(x.y1p, sc)), ca)),
                       ff_mul(x.y0p, sq)));
  hpi = ff_norm(ff_add(ff_mul(ff_norm(ff_mul(x.y2p, cb)), s2), ff_mul(ff_norm(ff_mul(x.y1p, sb)), sa)));
  hci = ff_norm(ff_add(ff_mul(ff_norm(ff_mul(x.y2m, cb)), c2), ff_mul(ff_norm(ff_mul(x.y1m, sb)), ca)));
  hcr = ff_norm(ff_neg(ff_add(ff_mul(ff_norm(ff_mul(x.y2m, uu)), s2), ff_mul(ff_norm(ff_mul(x.y1m, sc)), sa))));
}
// IMRPhenomPv2 bin: five sums per detector (mixed_bin_p's).
template <int NDET, class B>
GW_HD void acc_bin_p(const AccReq &x, B b, const AccTables &tb, const AccLut &lut, const ff4 *wd, const ff *w,
                     bool wshared, ff *acc) {
  const ff4 p = acc_ld(tb.pw + acc_at(b));
  const ff t{p.ch, p.cl};
  const ff a = acc_amp(x, b, t, ff{p.sh, p.sl}, lut);
  uint64_t al;
  const uint64_t ph = acc_offset(b) + acc_phase<true>(x, b, tb, lut, t, al);
  ff hpr, hpi, hcr, hci;
  acc_twist(x, b, tb, lut, t, al, hpr, hpi, hcr, hci);
  const ff aa = ff_norm(ff_sqr(a));
  const ff spp = ff_norm(ff_mul(aa, ff_norm(ff_add(ff_sqr(hpr), ff_sqr(hpi)))));
  const ff scc = ff_norm(ff_mul(aa, ff_norm(ff_add(ff_sqr(hcr), ff_sqr(hci)))));
  const ff spc = ff_norm(ff_mul(aa, ff_norm(ff_add(ff_mul(hpr, hcr), ff_mul(hpi, hci)))));
#pragma unroll
  for (int d = 0; d < NDET; d++) {
    ff c, s;
    ff_turns_sincos(ph + acc_linear(x, b, d), lut.turn, c, s);
    if (d == 0 || !wshared) {
      ff_acc(acc[kAccPerDet * d + 0], ff_mul(w[d], spp));
      ff_acc(acc[kAccPerDet * d + 1], ff_mul(w[d], scc));
      ff_acc(acc[kAccPerDet * d + 2], ff_mul(w[d], spc));
    }
    const ff dr{wd[d].ch, wd[d].cl}, di{wd[d].sh, wd[d].sl};
    const ff qr = ff_norm(ff_mul(a, ff_norm(ff_sub(ff_mul(dr, c), ff_mul(di, s)))));
    const ff qi = ff_norm(ff_mul(a, ff_norm(ff_add(ff_mul(dr, s), ff_mul(di, c)))));
    ff_acc(acc[kAccPerDet * d + 3], ff_add(ff_mul(qr, hpr), ff_mul(qi, hpi)));
    ff_acc(acc[kAccPerDet * d + 4], ff_add(ff_mul(qr, hcr), ff_mul(qi, hci)));
  }
}

// The model's polarisations / A_scale at bin n (zero beyond the cut): IMRPhenomD
// h+ = h (1 + cos^2 iota)/2 and hx = -i h cos iota are left to the caller as h;
// IMRPhenomPv2 h+, hx.
template <bool PV2>
GW_HD void acc_wave(const AccReq &x, int n, uint64_t qd, const AccTables &tb, const AccLut &lut, ff &pr, ff &pi,
                    ff &cr, ff &ci) {
  pr = pi = cr = ci = ff{0.f, 0.f};
  if (n > x.m.n_cut) return;
  AccBin b{n, qd};
  const ff4 p = acc_ld(tb.pw + n);
  const ff t{p.ch, p.cl};
  ff a = acc_amp(x, b, t, ff{p.sh, p.sl}, lut);
  a.h += x.bad;
  uint64_t al;
  const uint64_t ph = qd + acc_phase<PV2>(x, b, tb, lut, t, al) + x.B0 + x.B1 * (uint64_t)n;
  ff c, s;
  ff_turns_sincos(ph, lut.turn, c, s);
  const ff er = ff_norm(ff_mul(a, c)), ei = ff_norm(ff_neg(ff_mul(a, s)));  // a e^{-i psi}
  if constexpr (!PV2) {
    pr = er;
    pi = ei;
  } else {
    ff hpr, hpi, hcr, hci;
    acc_twist(x, b, tb, lut, t, al, hpr, hpi, hcr, hci);
    const ff tpr = ff_norm(ff_sub(ff_mul(hpr, er), ff_mul(hpi, ei))), tpi = ff_norm(ff_add(ff_mul(hpr, ei), ff_mul(hpi, er)));
    const ff txr = ff_norm(ff_sub(ff_mul(hcr, er), ff_mul(hci, ei))), txi = ff_norm(ff_add(ff_mul(hcr, ei), ff_mul(hci, er)));
    pr = ff_norm(ff_add(ff_mul(x.c2z, tpr), ff_mul(x.s2z, txr)));
    pi = ff_norm(ff_add(ff_mul(x.c2z, tpi), ff_mul(x.s2z, txi)));
    cr = ff_norm(ff_sub(ff_mul(x.c2z, txr), ff_mul(x.s2z, tpr)));
    ci = ff_norm(ff_sub(ff_mul(x.c2z, txi), ff_mul(x.s2z, tpi)));
  }
}

}  // namespace gwt

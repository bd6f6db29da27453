// two_float.h -- arithmetic on unevaluated sums of two FP32 numbers (48-bit
// significands), host and device.
//
// GB300 issues an FP32 instruction per sub-partition and cycle and an FP64
// instruction every 64 cycles, so an FP64-grade product or sum made of 4 to 11
// FP32 instructions is 6 to 16 times cheaper than the FP64 instruction.  The
// building blocks are Knuth's and Dekker's error-free sum and the product with
// its error from a fused multiply-add (Dekker, Numer. Math. 18 (1971); Knuth,
// TAOCP 2, 4.2.2).  A result carries a relative error of a few 2^-48, absolute
// to the larger operand where a sum cancels.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define TF_HD __host__ __device__ __forceinline__
#else
#define TF_HD inline
#endif

namespace gwt {

struct ff {
  float h, l;
};

// Single FP32 operations that the compiler may neither contract nor reorder.
#if defined(__CUDA_ARCH__)
TF_HD float f_add(float a, float b) { return __fadd_rn(a, b); }
TF_HD float f_sub(float a, float b) { return __fsub_rn(a, b); }
TF_HD float f_mul(float a, float b) { return __fmul_rn(a, b); }
TF_HD float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
TF_HD float f_rcp(float a) {  // within an ulp; callers correct it
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
TF_HD float f_rsqrt(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
TF_HD int f_bits(float a) { return __float_as_int(a); }
TF_HD float f_from_bits(int a) { return __int_as_float(a); }
TF_HD int f_to_int(float a) { return __float2int_rn(a); }
#else
TF_HD float f_add(float a, float b) { return a + b; }
TF_HD float f_sub(float a, float b) { return a - b; }
TF_HD float f_mul(float a, float b) { return a * b; }
TF_HD float f_fma(float a, float b, float c) { return std::fma(a, b, c); }
TF_HD float f_rcp(float a) { return 1.0f / a; }
TF_HD float f_rsqrt(float a) { return 1.0f / std::sqrt(a); }
TF_HD int f_bits(float a) {
  int i;
  std::memcpy(&i, &a, 4);
  return i;
}
TF_HD float f_from_bits(int a) {
  float f;
  std::memcpy(&f, &a, 4);
  return f;
}
TF_HD int f_to_int(float a) { return (int)std::lrintf(a); }
#endif

TF_HD ff ff_split(double v) {
  ff r;
  r.h = (float)v;
  r.l = (float)(v - (double)r.h);
  return r;
}
TF_HD double ff_value(ff a) { return (double)a.h + (double)a.l; }
TF_HD ff ff_neg(ff a) { return ff{-a.h, -a.l}; }
// a + b exactly
TF_HD ff two_sum(float a, float b) {
  const float s = f_add(a, b), t = f_sub(s, a);
  return ff{s, f_add(f_sub(a, f_sub(s, t)), f_sub(b, t))};
}
// a + b exactly for |a| >= |b| (or a = 0)
TF_HD ff quick_two_sum(float a, float b) {
  const float s = f_add(a, b);
  return ff{s, f_sub(b, f_sub(s, a))};
}
TF_HD ff two_prod(float a, float b) {
  const float p = f_mul(a, b);
  return ff{p, f_fma(a, b, -p)};
}
TF_HD ff ff_norm(ff a) { return quick_two_sum(a.h, a.l); }
// Products and sums without the closing normalisation: the low part may reach
// a few ulp of the high part (or its cancelled size), which the next operation
// takes as it is; ff_norm where a value is compared or its high part stands
// for it.
TF_HD ff ff_mul(ff a, ff b) {
  ff p = two_prod(a.h, b.h);
  p.l = f_fma(a.h, b.l, p.l);
  p.l = f_fma(a.l, b.h, p.l);
  return p;
}
TF_HD ff ff_mulf(ff a, float b) {
  ff p = two_prod(a.h, b);
  p.l = f_fma(a.l, b, p.l);
  return p;
}
TF_HD ff ff_sqr(ff a) {
  ff p = two_prod(a.h, a.h);
  p.l = f_fma(f_add(a.h, a.h), a.l, p.l);
  return p;
}
TF_HD ff ff_add(ff a, ff b) {
  ff s = two_sum(a.h, b.h);
  s.l = f_add(s.l, f_add(a.l, b.l));
  return s;
}
TF_HD ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }
TF_HD ff ff_addf(ff a, float b) {
  ff s = two_sum(a.h, b);
  s.l = f_add(s.l, a.l);
  return s;
}
// a / b: the quotient of the high parts and one correction.
TF_HD ff ff_div(ff a, ff b) {
  const float r = f_rcp(b.h), q = f_mul(a.h, r);
  float e = f_fma(-q, b.h, a.h);
  e = f_add(e, f_fma(-q, b.l, a.l));
  return quick_two_sum(q, f_mul(e, r));
}
// 1 / sqrt(a), a > 0: one Newton step with the residual 1 - a y^2 in two floats.
TF_HD ff ff_rsqrt(ff a) {
  const float y = f_rsqrt(a.h);
  const ff p = ff_mul(two_prod(y, y), a);
  const float e = f_sub(f_sub(1.0f, p.h), p.l);
  return quick_two_sum(y, f_mul(f_mul(0.5f, y), e));
}
// Running sum of two-float terms: the error of every addition is kept.
TF_HD void ff_acc(ff &s, ff v) {
  const ff t = two_sum(s.h, v.h);
  s.h = t.h;
  s.l = f_add(s.l, f_add(t.l, v.l));
}

// ---- turns: angles as 64-bit fixed point, 2^64 per turn ----
// A two-float number of turns, |a| < 2^21 -> fixed point, modulo one turn,
// with 2^-50 turn resolution.
TF_HD uint64_t ff_turns_q64(ff a) {
  const float big = 12582912.0f;  // 1.5 2^23: adding it rounds to an integer
  const float k = f_sub(f_add(a.h, big), big), r = f_sub(a.h, k);
  const float m = f_fma(r, 8388608.0f, big);
  const int i1 = f_bits(m) - 0x4B400000;  // r in 2^-23 turns
  const float rem = f_add(f_fma(f_sub(m, big), -1.0f / 8388608.0f, r), a.l);
  const int i2 = f_to_int(f_mul(rem, 1125899906842624.0f));  // 2^-50 turns; |rem| < 2^-21
  return ((uint64_t)(int64_t)i1 << 41) + ((uint64_t)(int64_t)i2 << 14);
}
// Cosine and sine of q / 2^64 turns from a table of kTurnTab (cos h, l, sin h, l)
// and the series of the remaining angle |d| <= pi / 512 (truncation below 1e-17):
// cos and sin within about 2e-15.
constexpr int kTurnTab = 512, kTurnBits = 9;
struct ff4 {
  float ch, cl, sh, sl;
};
TF_HD void ff_turns_sincos(uint64_t q, const ff4 *tab, ff &c, ff &s) {
  const uint32_t hi = (uint32_t)(q >> 32), lo = (uint32_t)q;
  const uint32_t idx = (hi + (1u << (31 - kTurnBits))) >> (32 - kTurnBits);
  const int rh = (int)(hi - (idx << (32 - kTurnBits)));  // |rh| <= 2^22
  // rh 2^-32 + lo 2^-64 turns in radians
  const float h = f_sub(f_from_bits(rh + 0x4B400000), 12582912.0f);
  const float l = f_sub(f_from_bits((int)(0x4B000000u | (lo >> 9))), 8388608.0f);  // lo in units of 2^-55
  const double wd = 6.28318530717958647692 / 4294967296.0;
  const float k1 = (float)wd, k2 = (float)(wd - (double)k1);
  const float dh = f_mul(h, k1);
  const float dl = f_fma(l, k1 * 1.1920928955078125e-07f, f_fma(h, k2, f_fma(h, k1, -dh)));
  // 1 - cos d = d^2/2 - d^4/24, sin d = d - d^3/6 + d^5/120
  const float d2 = f_mul(dh, dh);
  const float d2l = f_fma(f_add(dh, dh), dl, f_fma(dh, dh, -d2));
  const ff u{0.5f * d2, f_fma(f_mul(d2, d2), -1.0f / 24.0f, 0.5f * d2l)};
  const ff v{dh, f_fma(f_mul(dh, d2), f_fma(d2, 1.0f / 120.0f, -1.0f / 6.0f), dl)};
  const ff4 t = tab[idx & (kTurnTab - 1)];
  const ff C{t.ch, t.cl}, S{t.sh, t.sl};
  // cos: C - S v - C u; sin: S + C v - S u
  const ff sv = ff_mul(S, v), cu = ff_mul(C, u), cv = ff_mul(C, v), su = ff_mul(S, u);
  ff a = two_sum(C.h, -sv.h);
  ff b = two_sum(a.h, -cu.h);
  c = quick_two_sum(b.h, f_add(b.l, f_add(a.l, f_sub(C.l, f_add(sv.l, cu.l)))));
  a = two_sum(S.h, cv.h);
  b = two_sum(a.h, -su.h);
  s = quick_two_sum(b.h, f_add(b.l, f_add(a.l, f_add(S.l, f_sub(cv.l, su.l)))));
}
// exp(z), z normalised, from a table of 2^(j/64), j = 0..63 (zero below e^-87,
// infinite above e^88, as FP32).
constexpr int kExpTab = 64;
TF_HD ff ff_exp(ff z, const ff *tab) {
  const float big = 12582912.0f;
  if (!(z.h > -87.0f)) return z.h != z.h ? z : ff{0.0f, 0.0f};
  if (z.h > 88.0f) return ff{INFINITY, 0.0f};
  const double step = 0.69314718055994530942 / kExpTab;
  // step = c1 + c2 + c3 with 12 bits in c1: k c1 is exact for |k| < 2^12 .. 2^13
  const float c1 = (float)((int)(step * 262144.0)) / 262144.0f;
  const float c2 = (float)(step - (double)c1), c3 = (float)(step - (double)c1 - (double)c2);
  const float m = f_fma(z.h, (float)(kExpTab / 0.69314718055994530942), big);
  const int k = f_bits(m) - 0x4B400000;
  const float kf = f_sub(m, big);
  const float a = f_fma(-kf, c1, z.h);
  const ff p = two_prod(kf, c2);
  const ff r0 = two_sum(a, -p.h);
  const ff r = quick_two_sum(r0.h, f_add(f_sub(r0.l, p.l), f_fma(-kf, c3, z.l)));  // |r| < 0.0055
  const ff r2 = ff_sqr(r);
  const float hi3 = f_mul(f_mul(r2.h, r.h), f_fma(r.h, f_fma(r.h, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f));
  ff w = quick_two_sum(r.h, 0.5f * r2.h);
  w.l = f_add(w.l, f_add(f_fma(0.5f, r2.l, r.l), hi3));
  const ff T = tab[k & (kExpTab - 1)];
  const ff tw = ff_mul(T, w);
  ff e = quick_two_sum(T.h, tw.h);
  e.l = f_add(e.l, f_add(T.l, tw.l));
  const float sc = f_from_bits((127 + (k >> 6)) << 23);
  return ff{f_mul(e.h, sc), f_mul(e.l, sc)};
}
// atan(y) as a table angle and a remainder: i steps of 1 / kTurnTab turn
// (|i| <= kTurnTab / 4) plus d radians, |d| < 0.0063.
TF_HD int ff_atan(ff y, const ff4 *tab, ff &d) {
  const float ay = fabsf(y.h);
  const bool inv = ay > 1.0f;
  const float r = inv ? f_rcp(ay) : ay, r2 = r * r;
  // Abramowitz & Stegun 4.4.49 (1e-5): only picks the table angle
  const float p = r * f_fma(r2, f_fma(r2, f_fma(r2, f_fma(r2, 0.0208351f, -0.0851330f), 0.1801410f), -0.3302995f), 0.9998660f);
  int i = f_to_int(p * (float)(kTurnTab / 6.28318530717958647692));
  if (inv) i = kTurnTab / 4 - i;
  if (y.h < 0.0f) i = -i;
  const ff4 t = tab[i & (kTurnTab - 1)];
  const ff C{t.ch, t.cl}, S{t.sh, t.sl};
  // z = tan(atan y - theta) = (y C - S) / (C + y S)
  const ff num = ff_norm(ff_sub(ff_mul(y, C), S)), den = ff_norm(ff_add(C, ff_mul(y, S)));
  const ff z = ff_div(num, den);
  const float z2 = z.h * z.h;
  d = ff{z.h, f_fma(f_mul(z.h, z2), f_fma(z2, 0.2f, -1.0f / 3.0f), z.l)};
  return i;
}

// Host: the two tables.
inline void ff_fill_tables(ff4 *turn, ff *ex) {
  for (int i = 0; i < kTurnTab; i++) {
    // octant symmetry keeps the quarter turns exact
    const double th = 6.28318530717958647692 * i / kTurnTab;
    double c = std::cos(th), s = std::sin(th);
    if (i % (kTurnTab / 4) == 0) {
      c = i == 0 ? 1 : i == kTurnTab / 2 ? -1 : 0;
      s = i == kTurnTab / 4 ? 1 : i == 3 * kTurnTab / 4 ? -1 : 0;
    }
    const ff a = ff_split(c), b = ff_split(s);
    turn[i] = ff4{a.h, a.l, b.h, b.l};
  }
  for (int j = 0; j < kExpTab; j++) ex[j] = ff_split(std::exp2((double)j / kExpTab));
}

}  // namespace gwt

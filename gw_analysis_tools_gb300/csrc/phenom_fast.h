// phenom_fast.h -- the per-request prologue of the batched and plain forms in
// short, independent parts (host and device).
//
// The same constants as phenom_prologue.h (which the Fisher's difference
// quotients keep), arranged for latency: an FP64 instruction occupies a
// sub-partition's FP64 pipe for 64 cycles whatever the number of active lanes,
// so what counts is the number of FP64 instructions in a row.  Therefore
//  * the inspiral side of the amplitude and phase connections is evaluated at
//    M f = 0.014 and 0.018, numbers that no request changes: the powers and
//    logarithms there are literals;
//  * the intermediate amplitude is the quartic through its five conditions in
//    the variable centred between the matching frequencies (a dozen products)
//    instead of five closed expressions in powers of the frequencies;
//  * the calibration fits and the PN coefficients are rows of tables, so that
//    lanes evaluate different rows with the same instructions;
//  * every root, logarithm and reciprocal of M, f_ref and df is taken once
//    (those of df when the stream is registered), and (M f)^(i/3) are products;
//  * Pv2's rotations work on components: a sine and cosine of an angle that
//    was just taken from components is their ratio, and the time shift's
//    10-node spline derivative is a fixed combination of its node values.
// The parts are functions of their own (not inlined): every kernel that runs
// them, whatever its register bound, then gives the same bits, and the code
// stays small enough for the instruction caches.
#pragma once

#include "phenom_acc.h"

namespace gwt {

// Literals at M f = 0.018: powers of (pi 0.018)^(1/3), ln(pi 0.018), 0.018^(1/3), ln 0.018;
// the amplitude's sqrt(pi 40 / 192) pi^(-7/6) and sqrt(pi / 30) pi^(-7/6); the harmonics' roots.
constexpr double kFastV2 = 0.147326742094114666947;
constexpr double kFastV3 = 0.0565486677646162782923;
constexpr double kFastV4 = 0.0217051689360657785201;
constexpr double kFastV5 = 0.00833113099152339819391;
constexpr double kFastV6 = 0.0031977518259529521925;
constexpr double kFastV7 = 0.00122739838694045349123;
constexpr double kFastVm5 = 120.031722105613404997;
constexpr double kFastL = -2.8726536352365721857;
constexpr double kFastW = 0.262074139420889660714;
constexpr double kFastLx = -4.01738352108597235985;
constexpr double kFastAmp = 0.212787510139663399158;
constexpr double kFastAmpSky = 0.0851150040558653596631;
constexpr double kFastY2 = 0.157695782626260003015;
constexpr double kFastY1 = 0.315391565252520006031;
constexpr double kFastY0 = 0.386274202023189580342;

// What a grid's spacing contributes: df, 1/df, df^(1/3), ln df, df^(-7/6), df^(3/4).
struct GridConst {
  double df, idf, c13, ln, m76, q34;
};
inline GridConst grid_const(double df) {
  return GridConst{df, 1.0 / df, std::cbrt(df), std::log(df), std::pow(df, -7. / 6.), std::pow(df, 0.75)};
}

// Source quantities that every part starts from (recomputed by each warp).
struct FastCore {
  double m1, m2, M, iM, eta, ieta, delta, c1, c2, cs, ca, chi_pn;
};
// Intermediate values of one request between the parts.
struct FastX {
  double iM, delta, cM, lM, cfr, lfr, M34;  // M^(1/3), ln M, f_ref^(1/3), ln f_ref, M^(3/4)
  double xr, xd, x3, h;                     // ringdown, damping, peak in M f; half the intermediate range
  double v1, d1, v3, d3, ins1, dins1;       // connection values (derivatives by M f)
  double l2, i2, p2, y2, at2;               // at x2 = xr / 2: ln, 1/x2, x2^(3/4), atan argument and value
  double a[5];                              // intermediate amplitude in u = (M f - xm) / h
  double phi_fref;
  int have_phi, pad;
  double sn[5], cn[5];                      // of the hour angle, DEC, psi, inclination, phiRef
  double node[kPv2ShiftNodes];
};

GW_HDNI FastCore fast_core(const GenParams &in) {
  FastCore k;
  k.m1 = in.mass1 * kMsolSec;
  k.m2 = in.mass2 * kMsolSec;
  k.M = k.m1 + k.m2;
  k.iM = 1. / k.M;
  // eta and sqrt(1 - 4 eta) rounded as the reference's: near equal masses the
  // root shows the last bit of eta
  k.eta = (k.m1 * k.m2) / (k.M * k.M);
  k.ieta = 1. / k.eta;
  k.delta = sqrt(1. - 4 * k.eta);
  k.c1 = in.spin1[2];
  k.c2 = in.spin2[2];
  k.cs = 0.5 * (k.c1 + k.c2);
  k.ca = 0.5 * (k.c1 - k.c2);
  const double chi_eff = (k.m1 * k.c1 + k.m2 * k.c2) * k.iM;
  k.chi_pn = chi_eff - ((38. / 113) * k.eta) * (2 * k.cs);
  return k;
}
GW_HD void fast_store(Source &s, FastX &x, const GenParams &in, const FastCore &k) {
  s.mass1 = k.m1;
  s.mass2 = k.m2;
  s.spin1x = in.spin1[0];
  s.spin2x = in.spin2[0];
  s.spin1y = in.spin1[1];
  s.spin2y = in.spin2[1];
  s.spin1z = k.c1;
  s.spin2z = k.c2;
  s.chi_s = k.cs;
  s.chi_a = k.ca;
  s.eta = k.eta;
  s.inv_eta = k.ieta;
  s.k_tf2 = (3. / 128.) * k.ieta;
  s.M = k.M;
  s.chi_pn = k.chi_pn;
  s.DL = in.Luminosity_Distance * (kMpcSI / kC);
  s.delta_mass = k.delta;
  s.phiRef = in.phiRef;
  s.tc = in.tc;
  s.sky_average = in.sky_average;
  s.incl_angle = in.incl_angle;
  s.f_ref = in.f_ref;
  s.shift_time = in.shift_time;
  s.shift_phase = in.shift_phase;
  s.dep_postmerger = in.dep_postmerger;
  s.pv2 = 0;
  s.chip = in.chip;
  s.phip = in.phip;
  s.f1_phase = 0.018 * k.iM;
  s.f1 = 0.014 * k.iM;
  x.iM = k.iM;
  x.delta = k.delta;
}

// ---- tables by row ----
// PN coefficients: row = coefficient, columns = [1, d ca, cs, ca^2, d ca cs, cs^2] x [1, eta, eta^2, eta^3]
// (IMRPhenomD.cpp:955-1032; d = sqrt(1 - 4 eta)).  Rows: amplitude 2..6, phase 2, 3, 4, 7, 8, 10.
constexpr int kPnRows = 11, kPnMono = 6, kPnEta = 4;
#define GWT_PN_ROWS_INIT                                                                                              \
  {{{-323. / 224, 451. / 168}},                                                                                       \
   {{0}, {27. / 8}, {27. / 8, -11. / 6}},                                                                             \
   {{-27312085. / 8128512, -1975055. / 338688, 105271. / 24192}, {0}, {0}, {-81. / 32, 8}, {-81. / 16},               \
    {-81. / 32, 17. / 8}},                                                                                            \
   {{-85 * kPi / 64, 85 * kPi / 16}, {285197. / 16128, -1579. / 4032},                                                \
    {285197. / 16128, -15317. / 672, -2227. / 1008}},                                                                 \
   {{-177520268561. / 8583708672, 545384828789. / 5007163392 - 205 * kPi * kPi / 48, -3248849057. / 178827264,        \
     34473079. / 6386688},                                                                                            \
    {31 * kPi / 12},                                                                                                  \
    {31 * kPi / 12, -7 * kPi / 3},                                                                                    \
    {1614569. / 64512, -1873643. / 16128, 2167. / 42},                                                                \
    {1614569. / 32256, -165961. / 2688},                                                                              \
    {1614569. / 64512, -61391. / 1344, 57451. / 4032}},                                                               \
   {{3715. / 756, 55. / 9}},                                                                                          \
   {{-16. * kPi}, {113. / 3}, {113. / 3, -76. / 3}},                                                                  \
   {{15293365. / 508032, 27145. / 504, 3085. / 72}, {0}, {0}, {-405. / 8, 200.}, {-405. / 4}, {-405. / 8, 5. / 2}},   \
   {{77096675. * kPi / 254016, 378515. * kPi / 1512, -74045. * kPi / 756},                                            \
    {-25150083775. / 3048192, 26804935. / 6048, -1985. / 48},                                                         \
    {-25150083775. / 3048192, 10566655595. / 762048, -1042165. / 3024, 5345. / 36}},                                  \
   {{38645. * kPi / 756, -65. * kPi / 9}, {-732985. / 2268, -140. / 9}, {-732985. / 2268, 24260. / 81, 340. / 9}},    \
   {{11583231236531. / 4694215680 - 6848. * kGammaE / 21 - 640. * kPi * kPi / 3 - 6848. * kLog64 / 63,                \
     -15737765635. / 3048192 + 2255. * kPi * kPi / 12, 76055. / 1728, -127825. / 1296},                               \
    {2270. * kPi / 3},                                                                                                \
    {2270. * kPi / 3, -520. * kPi}}}
static const double gwt_pn_rows_h[kPnRows][kPnMono][kPnEta] = GWT_PN_ROWS_INIT;
#if defined(__CUDACC__)
// in global memory: lanes read different rows
static __device__ const double gwt_pn_rows_d[kPnRows][kPnMono][kPnEta] = GWT_PN_ROWS_INIT;
static __device__ const double gwt_fit_rows_d[19][11] = GWT_LAMBDA_FIT_INIT;
#endif
GW_HD const double *fast_fit_row(int i) {
#if defined(__CUDA_ARCH__)
  return gwt_fit_rows_d[i];
#else
  return gwt_lambda_fit_h[i];
#endif
}
GW_HDNI void fast_fit(Lambda &l, const FastCore &k, int i) {  // IMRPhenomD.cpp:855-870
  const double *p = fast_fit_row(i);
  const double e = k.eta, xi = k.chi_pn - 1;
  const double a = fma(e, p[1], p[0]), b = fma(e, fma(e, p[4], p[3]), p[2]), c = fma(e, fma(e, p[7], p[6]), p[5]),
               d = fma(e, fma(e, p[10], p[9]), p[8]);
  const double v = fma(xi, fma(xi, fma(xi, d, c), b), a);
  double *dst = i < 3 ? &l.rho[i] : i == 3 ? &l.v2 : i < 7 ? &l.gamma[i - 4] : i < 11 ? &l.sigma[i - 6]
              : i < 14 ? &l.beta[i - 10] : &l.alpha[i - 13];
  *dst = v;
}
GW_HDNI void fast_pn(ModelD &m, const FastCore &k, int i) {
#if defined(__CUDA_ARCH__)
  const double(*t)[kPnEta] = gwt_pn_rows_d[i];
#else
  const double(*t)[kPnEta] = gwt_pn_rows_h[i];
#endif
  const double da = k.delta * k.ca, mono[kPnMono] = {1.0, da, k.cs, k.ca * k.ca, da * k.cs, k.cs * k.cs};
  double v = 0.0;
#pragma unroll
  for (int j = kPnMono - 1; j >= 0; j--) {
    const double c = fma(k.eta, fma(k.eta, fma(k.eta, t[j][3], t[j][2]), t[j][1]), t[j][0]);
    v = fma(c, mono[j], v);
  }
  if (i < 5) {
    m.pn_amp[2 + i] = v;
  } else {
    const int q = i < 8 ? i - 3 : i < 10 ? i - 1 : 10;  // phase 2, 3, 4, 7, 8, 10
    m.pn_phase[q] = v;
    if (q == 8) m.pn_phase[9] = v;
  }
}
// The entries that no row sets.
GW_HD void fast_fixed(ModelD &m) {
  Lambda &l = m.l;
  l.rho[3] = l.gamma[3] = l.sigma[0] = l.beta[0] = l.beta[4] = l.alpha[0] = l.alpha[6] = 0;
  m.pn_amp[0] = 1.;
  m.pn_amp[1] = 0.;
  m.pn_phase[0] = 1.;
  m.pn_phase[1] = m.pn_phase[5] = m.pn_phase[6] = 0.;
  m.pn_phase[11] = 6848. / 63.;
  precalc_powers_PI(m.pi);
}

// ---- ringdown ----
GW_HD double fast_final_spin(double eta, double ieta, double delta, double chi1, double chi2) {  // IMRPhenomD.cpp:1229-1257
  const double m1 = 0.5 * (1.0 + delta), m2 = 0.5 * (1.0 - delta);
  const double s = m1 * m1 * chi1 + m2 * m2 * chi2;
  const double n0 = 3.4641016151377544 + eta * (-4.399247300629289 + eta * (9.397292189321194 - 13.180949901606242 * eta));
  const double n1 = ieta - 0.0850917821418767 - 5.837029316602263 * eta;
  const double n2 = 0.1014665242971878 - 2.0967746996832157 * eta;
  const double n3 = -1.3546806617824356 + 4.108962025369336 * eta;
  const double n4 = -0.8676969352555539 + 2.064046835273906 * eta;
  return eta * (n0 + s * (n1 + s * (n2 + s * (n3 + s * n4))));
}
// post_merger (IMRPhenomD.cpp:1091-1217): ringdown and damping frequencies.
// The radiated energy eta P (1 + A s) / (1 + B s), s = t / u, enters through
// 1 / (1 - E) alone: one division for both.
GW_HDNI void fast_ring(Source &s, FastX &x, const FastCore &k, const double *qnm) {
  if (s.dep_postmerger) {
    post_merger(s, qnm);
    x.xr = s.fRD * k.M;
    x.xd = s.fdamp * k.M;
    return;
  }
  double af;
  if (!s.pv2) {
    af = fast_final_spin(k.eta, k.ieta, k.delta, k.c1, k.c2);
  } else {  // IMRPhenomP.cpp:1232-1253
    const bool first = k.m1 >= k.m2;
    const double par = first ? fast_final_spin(k.eta, k.ieta, k.delta, k.c1, k.c2)
                             : fast_final_spin(k.eta, k.ieta, k.delta, k.c2, k.c1);
    const double qf = (first ? k.m1 : k.m2) * k.iM, sperp = s.chip * qf * qf;
    const double t = sqrt(sperp * sperp + par * par);
    // the reference's sign, sqrt(1 / par^2) par, is no number at par = 0
    af = par > 0 ? t : par < 0 ? -t : NAN;
  }
  const double m1 = 0.5 * (1.0 + k.delta), m2 = 0.5 * (1.0 - k.delta), w1 = m1 * m1, w2 = m2 * m2, e = k.eta;
  const double t = w1 * k.c1 + w2 * k.c2, u = w1 + w2;
  const double P = e * (0.055974469826360077 + e * (0.5809510763115132 + e * (-0.9606726679372312 + 3.352411249771192 * e)));
  const double A = -0.0030302335878845507 + e * (-2.0066110851351073 + 7.7050567802399215 * e);
  const double B = -0.6714403054720589 + e * (-1.4756929437702908 + 7.304676214885011 * e);
  const double den = u + B * t, sc = den / (den - P * (u + A * t));
  const double *a = qnm, *yr = qnm + kQnmLen, *yd = qnm + 2 * kQnmLen, *cr = qnm + 3 * kQnmLen,
               *cd = qnm + 4 * kQnmLen, *br = qnm + 5 * kQnmLen, *dr = qnm + 6 * kQnmLen, *bd = qnm + 7 * kQnmLen,
               *dd = qnm + 8 * kQnmLen;
  const int ilo = cspline_locate_near_uniform(a, kQnmLen, af, 0.002);
  x.xr = cspline_eval_pre(a, yr, br, cr, dr, ilo, af) * sc;
  x.xd = cspline_eval_pre(a, yd, bd, cd, dd, ilo, af) * sc;
  s.fRD = x.xr * k.iM;
  s.fdamp = x.xd * k.iM;
}
// Peak of the ringdown amplitude in M f (fpeak, IMRPhenomD.cpp:1312-1326) and
// its distance from the ringdown frequency in units of gamma3 fdamp.
GW_HD double fast_peak(const Lambda &l, const FastX &x, double &y) {
  const double g2 = l.gamma[1], w = x.xd * l.gamma[2];
  y = (g2 > 1 ? -1. : sqrt(1 - g2 * g2) - 1) / g2;
  const double v = x.xr + w * y;
  if (!(v < 0)) return v;
  y = (-v - x.xr) / w;  // the reference takes |v|
  return -v;
}
// Regions, and what makes the request invalid (model_d_freqs).
GW_HD void fast_freqs(ModelD &m, const FastX &x, double x3) {
  Source &s = m.s;
  s.f2_phase = 0.5 * s.fRD;
  s.f3 = x3 * x.iM;
  m.fcut = 0.2 * x.iM;
  m.status = kModelOK;
  if (!(s.eta > 0 && s.eta <= 0.25 + 1e-12) || !(s.fRD > 0) || !(s.fdamp > 0) || !(s.M > 0)) m.status |= kModelQnmRange;
}
// Ringdown amplitude and its derivative at the peak (IMRPhenomD.cpp:1468-1532).
GW_HDNI void fast_high(ModelD &m, FastX &x) {
  const Lambda &l = m.l;
  double y;
  x.x3 = fast_peak(l, x, y);
  x.h = 0.5 * (x.x3 - 0.014);
  fast_freqs(m, x, x.x3);
  const double iw = 1.0 / (l.gamma[2] * x.xd), q = 1.0 / (1.0 + y * y);
  x.v3 = l.gamma[0] * exp(-l.gamma[1] * y) * (iw * q);
  x.d3 = -x.v3 * iw * (l.gamma[1] + 2 * y * q);
}
// Inspiral amplitude and phase with their derivatives at M f = 0.014 and 0.018.
GW_HDNI void fast_low_amp(const ModelD &m, FastX &x) {
  // (pi 0.014)^(i/3), 0.014^((7 + i)/3)
  const double v2 = 0.12460016160013278761, v3 = 0.043982297150257105338, v4 = 0.015525200270779205274,
               v5 = 0.0054802013324670951107, v6 = 0.0019344424626135142893, r7 = 0.000047238788377834507728,
               r8 = 0.000011385220037784860011, r9 = 2.744e-6, i3 = 1.0 / (3 * 0.014);
  const double *p = m.pn_amp, *r = m.l.rho;
  const double t2 = p[2] * v2, t3 = p[3] * v3, t4 = p[4] * v4, t5 = p[5] * v5, t6 = p[6] * v6, u7 = r[0] * r7,
               u8 = r[1] * r8, u9 = r[2] * r9;
  x.v1 = 1.0 + t2 + t3 + t4 + t5 + t6 + u7 + u8 + u9;
  x.d1 = i3 * (2 * t2 + 3 * t3 + 4 * t4 + 5 * t5 + 6 * t6 + 7 * u7 + 8 * u8 + 9 * u9);
}
GW_HDNI void fast_low_phase(const ModelD &m, FastX &x) {
  // v = (pi 0.018)^(1/3): v^i, ln(pi 0.018), v^-5; w = 0.018^(1/3)
  constexpr double v2 = kFastV2, v3 = kFastV3, v4 = kFastV4, v5 = kFastV5, v6 = kFastV6, v7 = kFastV7, L = kFastL,
                   vm5 = kFastVm5, w = kFastW, xx = 0.018, ix = 1.0 / 0.018, i3 = 1.0 / (3 * 0.018);
  const double *p = m.pn_phase, *g = m.l.sigma;
  const double K = m.s.k_tf2 * vm5;
  const double t2 = p[2] * v2, t3 = p[3] * v3, t4 = p[4] * v4, t5 = (p[8] + p[9] * L) * v5,
               t6 = (p[10] - p[11] * L) * v6, t7 = p[7] * v7;
  const double S = 1.0 + t2 + t3 + t4 + t5 + t6 + t7;
  const double dS = i3 * (2 * t2 + 3 * t3 + 4 * t4 + 5 * t5 + 6 * t6 + 7 * t7) + ix * (p[9] * v5 - p[11] * v6);
  const double n = g[1] * xx + (0.75 * xx * w) * g[2] + (0.6 * xx * w * w) * g[3] + (0.5 * xx * xx) * g[4];
  const double dn = g[1] + g[2] * w + g[3] * (w * w) + g[4] * xx;
  x.ins1 = -kPi / 4. + K * S + m.s.inv_eta * n;
  x.dins1 = K * (dS - (5. * i3) * S) + m.s.inv_eta * dn;
}
// Intermediate and ringdown phase terms at x2 = xr / 2.
GW_HDNI void fast_f2_powers(FastX &x) {
  const double x2 = 0.5 * x.xr;
  x.l2 = log(x2);
  x.i2 = 1. / x2;
  x.p2 = sqrt(x2 * sqrt(x2));
}
GW_HDNI void fast_f2_atan(const ModelD &m, FastX &x) {
  x.y2 = (0.5 - m.l.alpha[5]) * x.xr / x.xd;
  x.at2 = atan(x.y2);
}
// Phase at f_ref when it lies in the inspiral (have_phi).
GW_HDNI void fast_fref_phase(const ModelD &m, FastX &x) {
  const Source &s = m.s;
  x.have_phi = 0;
  if (s.pv2 || !s.shift_phase || !(s.f_ref < s.f1_phase)) return;
  const double w = x.cM * x.cfr, v = m.pi.PIthird * w, L = kLnPi + x.lM + x.lfr, xf = w * w * w;
  const double *p = m.pn_phase, *g = m.l.sigma;
  const double c5 = p[8] + p[9] * L, c6 = p[10] - p[11] * L, v2 = v * v;
  const double S = 1.0 + v2 * (p[2] + v * (p[3] + v * (p[4] + v * (c5 + v * (c6 + v * p[7])))));
  const double n = xf * (g[1] + w * (0.75 * g[2] + w * (0.6 * g[3] + w * (0.5 * g[4]))));
  x.phi_fref = -kPi / 4. + s.k_tf2 * S / (v2 * v2 * v) + s.inv_eta * n;
  x.have_phi = 1;
}
// D: the time shift, the ringdown phase's derivative at the peak with the fit
// of alpha1 (IMRPhenomD.cpp:434-470; sets m.tcs in radians per Hz).  Call
// before fast_connect replaces alpha1.
GW_HDNI void fast_time_shift(ModelD &m, const FastX &x) {
  const Source &s = m.s;
  const Lambda &l = m.l;
  m.tcs = 0.0;
  if (!s.shift_time) return;
  double y3;
  const double x3 = fast_peak(l, x, y3), ix3 = 1. / x3, q = x3 - l.alpha[5] * x.xr;
  const double x3m14 = sqrt(sqrt(ix3));
  const double at = l.alpha[4] * x.xd / (x.xd * x.xd + q * q);
  m.tcs = s.M * s.inv_eta * (at + l.alpha[2] * (ix3 * ix3) + l.alpha[1] + l.alpha[3] * x3m14);
}
// C1 connections (IMRPhenomD.cpp:1614-1674), all in M f.
GW_HDNI void fast_connect(ModelD &m, const FastX &x) {
  Lambda &l = m.l;
  const double eta = m.s.eta;
  constexpr double x1 = 0.018, ix1 = 1.0 / 0.018, l1 = kFastLx;
  const double b2 = l.beta[2], b3 = l.beta[3];
  const double b1 = eta * x.dins1 - (b2 * ix1 + b3 * (ix1 * ix1 * ix1 * ix1));
  const double b0 = eta * x.ins1 - (b1 * x1 + b2 * l1 - b3 * (ix1 * ix1 * ix1 / 3.));
  const double x2 = 0.5 * x.xr, i2 = x.i2, i2_3 = i2 * i2 * i2;
  const double dint = b1 + b2 * i2 + b3 * (i2_3 * i2);
  const double dmr = l.alpha[2] * (i2 * i2) + l.alpha[3] * (x.p2 * i2) + l.alpha[4] / (x.xd * (1. + x.y2 * x.y2));
  const double a1 = dint - dmr;
  const double iv = b0 + b1 * x2 + b2 * x.l2 - b3 * (i2_3 * (1. / 3.));
  const double mr = a1 * x2 - l.alpha[2] * i2 + (4. / 3) * l.alpha[3] * x.p2 + l.alpha[4] * x.at2;
  l.beta[1] = b1;
  l.beta[0] = b0;
  l.alpha[1] = a1;
  l.alpha[0] = iv - mr;
}
// Linear phase constants (IMRPhenomD.cpp:434-470), after fast_time_shift and
// fast_fref_phase.  False when the phase at f_ref lies past the inspiral: then
// fast_finish_late after fast_connect.
GW_HDNI bool fast_finish_d(ModelD &m, const FastX &x) {
  const Source &s = m.s;
  m.tcl = 2 * kPi * s.tc + m.tcs;
  m.fref = s.shift_phase ? s.f_ref : 0;
  m.phic = s.shift_phase ? 2 * s.phiRef + x.phi_fref : s.phiRef;
  return !s.shift_phase || x.have_phi;
}
GW_HDNI void fast_finish_late(ModelD &m) {
  Pows pw;
  precalc_powers_ins(m.fref, m.s.M, pw);
  double pn[12];
  for (int j = 0; j < 12; j++) pn[j] = m.pn_phase[j];
  m.phic = 2 * m.s.phiRef + build_phase(m.fref, m, pn, pw);
}
// The intermediate amplitude through (v1, d1) at x1, v2 in the middle, (v3, d3)
// at x3: a quartic in u = (M f - xm) / h on [-1, 1].
GW_HDNI void fast_quartic(const ModelD &m, FastX &x) {
  const double D1 = x.d1 * x.h, D3 = x.d3 * x.h;
  const double s = 0.5 * (x.v3 + x.v1), d = 0.5 * (x.v3 - x.v1), ds = 0.5 * (D3 + D1), dd = 0.5 * (D3 - D1);
  const double e = s - m.l.v2;  // a2 + a4
  x.a[0] = m.l.v2;
  x.a[4] = 0.5 * dd - e;
  x.a[2] = e - x.a[4];
  x.a[3] = 0.5 * (ds - d);
  x.a[1] = d - x.a[3];
}
// p(u) = sum a_j u^j as coefficients of powers of t, u = t c + b.
GW_HD void fast_shift_quartic(const double *a, double c, double b, double *e) {
  double q[5];
  for (int j = 0; j < 5; j++) q[j] = a[j];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 3; j >= i; j--) q[j] = fma(q[j + 1], b, q[j]);
  double p = 1.0;
#pragma unroll
  for (int j = 0; j < 5; j++) {
    e[j] = q[j] * p;
    p *= c;
  }
}
// The quartic's coefficients in M f (Request's deltas; the FP64 bins' form).
GW_HDNI void fast_deltas(ModelD &m, const FastX &x) {
  const double ih = 1.0 / x.h;
  fast_shift_quartic(x.a, ih, -(0.014 + x.h) * ih, m.deltas);
}
// Amplitude normalisation (util.cpp:1271-1279) and its part in the bins'
// scale: A0 = c mc^(5/6) / D_L, mc^(5/6) = M^(5/6) eta^(1/2); A0eff = A0 M^(7/6).
GW_HDNI void fast_amp0(ModelD &m, const FastX &x, const GenParams &in, const FastCore &k) {
  const double c = (in.sky_average ? kFastAmpSky : kFastAmp), s6 = sqrt(x.cM);
  m.s.A0 = c * (x.cM * x.cM) * s6 * sqrt(k.eta) / (in.Luminosity_Distance * (kMpcSI / kC));
  m.A0eff = m.s.A0 * k.M * s6;
}

// ---- IMRPhenomPv2 ----
// chi_p and the in-plane angular momenta (PhenomPv2_Param_Transform,
// IMRPhenomP.cpp:1082-1210; reduced: :822-938), before the ringdown part.
GW_HDNI void fast_pv2_spins(Source &s, const GenParams &in, const FastCore &k) {
  s.pv2 = 1;
  const double q = k.m1 / k.m2;
  s.q = q;
  s.chil = (1.0 + q) / q * ((k.m1 * k.c1 + k.m2 * k.c2) * k.iM);
  if (!((in.chip + 1) > kCompThresh)) {
    const double m1_2 = k.m1 * k.m1, m2_2 = k.m2 * k.m2;
    const double S1 = m1_2 * sqrt(s.spin1y * s.spin1y + s.spin1x * s.spin1x);
    const double S2 = m2_2 * sqrt(s.spin2y * s.spin2y + s.spin2x * s.spin2x);
    const double A1 = 2 + 1.5 / q, A2 = 2 + 1.5 * q;
    const double a1 = A1 * S1, a2 = A2 * S2;
    s.chip = (a2 > a1 ? a2 : a1) / (k.m2 > k.m1 ? A2 * m2_2 : A1 * m1_2);
  } else {
    s.chip = in.chip;
    s.phip = in.phip;
  }
  const double f1 = k.m1 * k.iM, f2 = k.m2 * k.iM;
  s.SP = s.chip * f1 * f1;
  s.SL = k.c1 * f1 * f1 + k.c2 * f2 * f2;
}
// The J frame (IMRPhenomP.cpp:1130-1210): rotations by -phi_J about z, -theta_J
// about y and kappa about z, their sines and cosines from the components that
// define the angles.  sn/cn: of the inclination [3] and phiRef [4].
GW_HDNI void fast_pv2_frame(Source &s, ModelP &pm, const GenParams &in, const FastX &x) {
  const double m1_2 = s.mass1 * s.mass1, m2_2 = s.mass2 * s.mass2;
  const double v = 1.4645918875615231 * (x.cM * x.cfr), v2 = v * v, eta = s.eta;  // (pi M f_ref)^(1/3)
  const double L0 = s.M * s.M * (eta * (1.0 + (1.5 + eta / 6.0) * v2 + (3.375 - (19.0 * eta) / 8. - eta * eta / 24.0) * (v2 * v2))) / v;
  double Jx, Jy;
  if (!((in.chip + 1) > kCompThresh)) {
    Jx = m1_2 * s.spin1x + m2_2 * s.spin2x;
    Jy = m1_2 * s.spin1y + m2_2 * s.spin2y;
  } else {
    double sp, cp;
    sincos(s.phip, &sp, &cp);
    Jx = m1_2 * s.chip * cp;
    Jy = m1_2 * s.chip * sp;
  }
  const double Jz = L0 + m1_2 * s.spin1z + m2_2 * s.spin2z;
  const double p2 = Jx * Jx + Jy * Jy, p = sqrt(p2), iJ = 1.0 / sqrt(p2 + Jz * Jz);
  double cA = 1.0, sA = 0.0;
  s.phi_aligned = 0.0;
  if (p2 > 0) {
    const double ip = 1.0 / p;
    cA = Jx * ip;
    sA = -Jy * ip;
    s.phi_aligned = -atan2(Jy, Jx);
  }
  const double cB = Jz * iJ, sB = -p * iJ;
  const double si = x.sn[3], ci = x.cn[3], sr = x.sn[4], cr = x.cn[4];
  // N = (si cos(pi/2 - phiRef), si sin(pi/2 - phiRef), ci) through A and B
  double tx = si * sr, ty = si * cr, t1 = tx * cA - ty * sA;
  double ny = tx * sA + ty * cA;
  double nx = t1 * cB + ci * sB, nz = -t1 * sB + ci * cB;
  const double r2 = nx * nx + ny * ny;
  double cK = 1.0, sK = 0.0, r = 0.0;
  if (r2 > 0) {
    const double ir = 1.0 / sqrt(r2);
    r = r2 * ir;
    cK = nx * ir;
    sK = -ny * ir;
  }
  // L = z through A, B and K: its azimuth
  s.alpha0 = atan2(sB * sK, sB * cK);
  // X through A, B and K
  tx = -ci * sr;
  ty = -ci * cr;
  t1 = tx * cA - ty * sA;
  const double xy = tx * sA + ty * cA, xx = t1 * cB + si * sB, xz = -t1 * sB + si * cB;
  const double px = xx * cK - xy * sK, py = xx * sK + xy * cK;
  // zeta = atan2(X . Q, X . P), P = -y, Q = (Nz, 0, -Nx): cos and sin of 2 zeta
  const double P = -py, Q = px * nz - xz * r, n2 = P * P + Q * Q;
  pm.c2z = 1.0;
  pm.s2z = 0.0;
  if (n2 > 0) {
    const double in2 = 1.0 / n2;
    pm.c2z = (P * P - Q * Q) * in2;
    pm.s2z = 2.0 * P * Q * in2;
  }
  // s = -2, l = 2 harmonics at theta_JN: cos = Nz, sin = r (util.cpp:1953-2333)
  const double ct = nz, st = r;
  pm.Y[0] = kFastY2 * (1.0 - ct) * (1.0 - ct);
  pm.Y[1] = kFastY1 * st * (1.0 - ct);
  pm.Y[2] = kFastY0 * st * st;
  pm.Y[3] = kFastY1 * st * (1.0 + ct);
  pm.Y[4] = kFastY2 * (1.0 + ct) * (1.0 + ct);
}
// The constants at f_ref (model_p_finish), after the frame and the Euler angle
// coefficients (pv2_euler_coeffs).
GW_HDNI void fast_pv2_finish(ModelD &m, ModelP &pm, const FastX &x) {
  const Source &s = m.s;
  m.fref = s.f_ref;
  m.phic = 2 * s.phi_aligned;
  m.tcs = 0.0;
  m.tcl = 2 * kPi * s.tc;
  m.A0eff = m.A0eff / (2. * sqrt(5. / (64. * kPi)));
  const double v = 1.4645918875615231 * (x.cM * x.cfr), iv = 1.0 / v, l = kLnPi + x.lM + x.lfr;
  const double *a = pm.ac, *e = pm.ec;
  pm.alpha_shift = s.alpha0 - (iv * (a[2] + iv * (a[1] + iv * a[0])) + a[3] * l + a[4] * v);
  pm.eps_off = iv * (e[2] + iv * (e[1] + iv * e[0])) + e[3] * l + e[4] * v;
  if (!(s.f_ref > 0)) m.status |= kModelBadInput;
}
// Node j of the time shift (IMRPhenomP.cpp:551-606): the ringdown phase (times
// eta) at 0.8 .. 1.2 fRD without the terms linear in f.
GW_HDNI double fast_pv2_node(const ModelD &m, const FastX &x, int j) {
  const Lambda &l = m.l;
  const double rel = 0.8 + j * (0.4 / (kPv2ShiftNodes - 1)), xj = rel * x.xr;
  return -l.alpha[2] / xj + (4. / 3) * l.alpha[3] * sqrt(xj * sqrt(xj)) +
         l.alpha[4] * atan((xj - l.alpha[5] * x.xr) / x.xd);
}
// The natural spline's slope halfway between the middle ones of ten even
// nodes: sum_k w_k (y_(5+k) - y_(4-k)) / spacing (exact for linear terms).
GW_HDNI double fast_pv2_time_shift(const ModelD &m, const FastX &x) {
  const double w[5] = {1.2990196078431372549, -0.14705882352941176471, 0.039215686274509803922,
                       -0.0098039215686274509804, 0.0016339869281045751634};
  if (!m.s.shift_time || !(x.xr > 0)) return 0.0;
  double t = 0.0;
  for (int k = 0; k < 5; k++) t += w[k] * (x.node[5 + k] - x.node[4 - k]);
  const double slope = m.l.alpha[1] + t * ((kPv2ShiftNodes - 1) / 0.4) / x.xr;
  return -(m.s.inv_eta * m.s.M * slope) * (1.0 / (2. * kPi));
}

// ---- the grid's coefficients (mixed_phase_coeffs, mixed_amp_coeffs, mixed_regions) ----
GW_HDNI void fast_phase_coeffs(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o) {
  const Source &s = m.s;
  const Lambda &l = m.l;
  const double Mdf = s.M * g.df, iMdf = x.iM * g.idf, cu = x.cM * g.c13, Lx = x.lM + g.ln, Lc = kLnPi + Lx;
  const double K = s.k_tf2 * m.pi.PIminus_5third, *pn = m.pn_phase;
  const double icu2 = (cu * iMdf) * (cu * iMdf) * (cu * cu);  // cu^-2
  const double icu = cu * icu2;
  double q[12];
  q[0] = K;
  q[1] = 0.0;
  q[2] = (K * m.pi.PI2third) * pn[2];
  q[3] = (K * kPi) * pn[3];
  q[4] = (K * m.pi.PI4third) * pn[4];
  q[5] = (K * m.pi.PI5third) * (pn[8] + pn[9] * Lc) - kPi / 4.;
  q[6] = (K * m.pi.PIsquare) * (pn[10] - pn[11] * Lc);
  q[7] = (K * m.pi.PI7third) * pn[7];
  q[8] = l.sigma[1] * s.inv_eta;
  q[9] = (3. / 4.) * l.sigma[2] * s.inv_eta;
  q[10] = (3. / 5.) * l.sigma[3] * s.inv_eta;
  q[11] = (1. / 2.) * l.sigma[4] * s.inv_eta;
  double cp = icu2 * icu2 * icu;  // cu^-5
#pragma unroll
  for (int j = 0; j < 12; j++) {
    o.qi[j] = q[j] * cp;
    cp *= cu;
  }
  o.bi0 = K * m.pi.PI5third * pn[9];
  o.bi1 = -(K * m.pi.PIsquare) * pn[11] * cu;
  o.pA = (l.beta[0] + l.beta[2] * Lx) * s.inv_eta;
  o.pB = l.beta[1] * Mdf * s.inv_eta;
  o.pC = l.beta[2] * s.inv_eta;
  o.pD = l.beta[3] * s.inv_eta * ((1. / 3.) * (iMdf * iMdf * iMdf));
  o.mA = l.alpha[0] * s.inv_eta;
  o.mB = l.alpha[1] * Mdf * s.inv_eta;
  o.mC = l.alpha[2] * s.inv_eta * iMdf;
  o.mD = (4. / 3.) * l.alpha[3] * (x.M34 * g.q34) * s.inv_eta;
  o.mE = l.alpha[4] * s.inv_eta;
  o.mEq = (float)(o.mE * (1.0 / (2.0 * 3.14159265358979323846)) * kSegFScale);
  const double nc = l.alpha[5] * s.fRD * g.idf, nci = floor(nc);
  o.n_c = (int)nci;
  o.ncfrac = (float)(nc - nci);
  o.inv_nw = (float)(g.df / s.fdamp);
}
GW_HDNI void fast_amp_coeffs(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o) {
  const double cu = x.cM * g.c13, *pa = m.pn_amp;
  const double a[10] = {1.0,
                        0.0,
                        pa[2] * m.pi.PI2third,
                        pa[3] * kPi,
                        pa[4] * m.pi.PI4third,
                        pa[5] * m.pi.PI5third,
                        pa[6] * m.pi.PIsquare,
                        m.l.rho[0],
                        m.l.rho[1],
                        m.l.rho[2]};
  double c = 1.0;
#pragma unroll
  for (int j = 0; j < 10; j++) {
    split_f(a[j] * c, o.ai[j], o.ai_lo[j]);
    c *= cu;
  }
  // u = (n - n_m) Mdf / h, n_m the middle of the range in bins
  const double nm = 0.5 * (m.s.f1 + m.s.f3) * g.idf, nmid = floor(nm);
  o.n_mid = (int)nmid;
  const double ih = 1.0 / x.h, sc = m.s.M * g.df * ih;
  double e[5];
  fast_shift_quartic(x.a, sc, (nmid - nm) * sc, e);
#pragma unroll
  for (int j = 0; j < 5; j++) split_f(e[j], o.ei[j], o.ei_lo[j]);
  const double g1 = m.l.gamma[0], g2 = m.l.gamma[1], nrd = m.s.fRD * g.idf, nrdi = floor(nrd);
  o.n_rd = (int)nrdi;
  o.mrRDfrac = (float)(nrd - nrdi);
  const double w = m.l.gamma[2] * m.s.fdamp * g.idf;  // in bins
  split_f(g1 * w * (x.iM * g.idf), o.mrK, o.mrK_lo);
  split_f(g2 / w, o.mrExp, o.mrExp_lo);
  split_f(w * w, o.mrG2, o.mrG2_lo);
}
// grid_first from a product instead of a quotient: its correction steps find
// the same bin.
GW_HD int fast_grid_first(double fb, const GridConst &g, bool strict) {
  const double q = ceil(fb * g.idf);
  if (!(q < 2.0e9)) return 2000000000;
  int n = q > 0 ? (int)q : 0;
  auto ok = [&](int j) { return strict ? (double)j * g.df > fb : (double)j * g.df >= fb; };
  for (int it = 0; it < 4 && n > 0 && ok(n - 1); it++) n--;
  for (int it = 0; it < 4 && !ok(n) && n < 2000000000; it++) n++;
  return n;
}
GW_HDNI void fast_regions(const Request &r, const GridConst &g, MixedReq &o) {
  const ModelD &m = r.m;
  const Source &s = m.s;
  o.approximant = r.approximant;
  o.status = m.status;
  o.ndet = r.ndet;
  o.n_f1 = fast_grid_first(s.f1, g, false);
  o.n_f1p = fast_grid_first(s.f1_phase, g, false);
  o.n_f3 = fast_grid_first(s.f3, g, true);
  o.n_f2p = fast_grid_first(s.f2_phase, g, true);
  o.n_cut = fast_grid_first(m.fcut, g, true) - 1;
}
// A0eff (M df)^(-7/6) [times 1/2 for Pv2]: the powers of M cancel.
GW_HDNI double fast_a_scale(const Request &r, const GridConst &g) {
  const double a = r.m.s.A0 * g.m76;
  return r.approximant == kPhenomPv2 ? a * (0.5 / (2. * kFastY2)) : a;
}
GW_HDNI void fast_pv2_coeffs(const Request &r, const FastX &x, const GridConst &g, MixedReq &o) {
  const Source &s = r.m.s;
  const double eta = s.eta, cw = 1.4645918875615231 * (x.cM * g.c13), icw = 1.0 / cw, Lw = kLnPi + x.lM + g.ln;
  const double *a = r.p.ac, *e = r.p.ec;
  o.ea[0] = a[0] * (icw * icw * icw);
  o.ea[1] = a[1] * (icw * icw);
  o.ea[2] = a[2] * icw;
  o.ea[3] = a[3] * Lw + r.p.alpha_shift;
  o.ea[4] = a[4] * cw;
  o.ea[5] = a[3];
  o.ee[0] = e[0] * (icw * icw * icw);
  o.ee[1] = e[1] * (icw * icw);
  o.ee[2] = e[2] * icw;
  o.ee[3] = e[3] * Lw - r.p.eps_off;
  o.ee[4] = e[4] * cw;
  o.ee[5] = e[3];
#pragma unroll
  for (int k = 0; k < 5; k++) split_f(r.p.Y[k], o.Y[k], o.Y_lo[k]);
  const double l1 = 1.5 + eta / 6.0, l2 = 3.375 - (19.0 * eta) / 8. - eta * eta / 24.0, iSP = 1.0 / s.SP, w = eta * iSP;
  split_f(w, o.w[0], o.w_lo[0]);
  split_f(w * l1, o.w[1], o.w_lo[1]);
  split_f(w * l2, o.w[2], o.w_lo[2]);
  split_f(s.SL * iSP, o.w[3], o.w_lo[3]);
  split_f(cw * cw, o.x2c, o.x2c_lo);
}

// Detectors d0, d0 + step, ...: projections, phases; the finalize factors.
GW_HDNI void fast_antenna(Request &r, const FastX &x, const int *dets, int d0, int step) {
  const SkyTrig t{x.cn[0], x.sn[0], x.cn[1], x.sn[1], x.cn[2], x.sn[2]};
  for (int d = d0; d < r.ndet && d < kMaxDet; d += step) {
    antenna_trig(dets[d], t, r.det[d].fp, r.det[d].fc);
    r.det[d].tau = -dtoa_trig(t, dets[0], dets[d]) * (2 * kPi);
  }
}
GW_HDNI void fast_det_phase(const Request &r, double df, MixedReq &o, int d0, int step) {
  mixed_det_phase(r, df, o, d0, step);
}
GW_HDNI void fast_det_phase(const Request &r, double df, AccReq &o, int d0, int step) {
  acc_det_phase(r, df, o, d0, step);
}
GW_HDNI void fast_det_factors(const Request &r, MixedReq &o, const double *dscale, const double *wscale) {
  mixed_det_factors(r, o, dscale, wscale);
}

// The parts in order (host): request_prologue and the form's coefficients.
inline int fast_request(Request &r, FastX &x, const GenParams &in, int approximant, const int *dets, int ndet,
                        const double *qnm) {
  r.approximant = approximant;
  r.ndet = ndet;
  const bool pv2 = approximant == kPhenomPv2;
  const FastCore k = fast_core(in);
  ModelD &m = r.m;
  fast_store(m.s, x, in, k);
  fast_fixed(m);
  for (int i = 0; i < 19; i++) fast_fit(m.l, k, i);
  for (int i = 0; i < kPnRows; i++) fast_pn(m, k, i);
  const double ang[5] = {in.gmst - in.RA, in.DEC, in.psi, in.incl_angle, in.phiRef};
  for (int i = 0; i < (pv2 ? 5 : 4); i++) sincos(ang[i], &x.sn[i], &x.cn[i]);
  m.s.cos_incl = x.cn[3];
  m.s.fac_incl = .5 * (1 + x.cn[3] * x.cn[3]);
  x.cM = cbrt(k.M);
  x.lM = log(k.M);
  x.cfr = cbrt(in.f_ref);
  x.lfr = log(in.f_ref);
  x.M34 = sqrt(k.M * sqrt(k.M));
  fast_amp0(m, x, in, k);
  if (pv2) fast_pv2_spins(m.s, in, k);
  fast_ring(m.s, x, k, qnm);
  fast_high(m, x);
  fast_low_amp(m, x);
  fast_low_phase(m, x);
  fast_f2_powers(x);
  fast_f2_atan(m, x);
  fast_fref_phase(m, x);
  if (pv2) {
    fast_pv2_frame(m.s, r.p, in, x);
    pv2_euler_coeffs(r.p.ac, r.p.ec, m.s);
    fast_pv2_finish(m, r.p, x);
  } else {
    fast_time_shift(m, x);
  }
  fast_connect(m, x);
  fast_quartic(m, x);
  fast_deltas(m, x);
  if (pv2) {
    for (int j = 0; j < kPv2ShiftNodes; j++) x.node[j] = fast_pv2_node(m, x, j);
    r.p.t_corr = fast_pv2_time_shift(m, x);
  } else if (!fast_finish_d(m, x)) {
    fast_finish_late(m);
  }
  fast_antenna(r, x, dets, 0, 1);
  return m.status;
}
inline int fast_acc(const Request &r, const FastX &x, const GridConst &g, AccReq &o, const double *dscale,
                    const double *wscale) {
  fast_regions(r, g, o.m);
  o.m.A_scale = fast_a_scale(r, g);
  fast_phase_coeffs(r.m, x, g, o.m);
  fast_amp_coeffs(r.m, x, g, o.m);
  if (r.approximant == kPhenomPv2) fast_pv2_coeffs(r, x, g, o.m);
  mixed_det_factors(r, o.m, dscale, wscale);
  acc_det_phase(r, g.df, o);
  acc_phase_coeffs(r, g.df, o);
  acc_amp_coeffs(r, g.df, o);
  if (r.approximant == kPhenomPv2) acc_pv2_coeffs(r, g.df, o);
  acc_range(r, o);
  return o.m.status;
}

}  // namespace gwt

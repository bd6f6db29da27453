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

// Literals: ln 0.018, (pi 0.018)^(1/3), (pi 0.2)^(1/3), 0.2^(3/4); the amplitude's
// sqrt(pi 40 / 192) pi^(-7/6) and sqrt(pi / 30) pi^(-7/6); the harmonics' roots.
constexpr double kFastLx = -4.01738352108597235985;
constexpr double kFastV = 0.383831658535502601325;
constexpr double kFastVc = 0.85649853169451150001;
constexpr double kFast34 = 0.299069756244244108382;
constexpr double kFastAmp = 0.212787510139663399158;
constexpr double kFastAmpSky = 0.0851150040558653596631;
constexpr double kFastY2 = 0.157695782626260003015;
constexpr double kFastY1 = 0.315391565252520006031;
constexpr double kFastY0 = 0.386274202023189580342;
// Rows of fast_low: coefficients of the PN terms and fits at M f = 0.014 (rows 0,
// 1) and 0.018 (rows 2, 3: those of the series times (pi M f)^(-5/3), ln(pi M f)
// inside), then the constant; the time shift's nodes at 2 rel = M f / (xr / 2).
#define GWT_LOW_ROWS_LITERALS \
  {{0.124600161600132787606, 0.0439822971502571053385, 0.0155252002707792052744, 0.00548020133246709511068, 0.00193444246261351428929, 0.0, 0.0000472387883778345077281, 0.0000113852200377848600105, 0.000002744, 0.0, 1.0}, \
   {5.93334102857775179078, 3.14159265358979323846, 1.4785905019789719309, 0.652404920531797036986, 0.276348923230502041327, 0.0, 0.00787313139630575128802, 0.00216861334053044952582, 0.000588, 0.0, 0.0}, \
   {17.6838825657661484188, 6.78763397456507990334, 2.60530880598924009842, 0.147326742094114666947, -1.8726536352365721857, 0.383831658535502601325, 0.018, 0.00353800088218201041964, 0.00074177482917455905034, 0.000162, 239.884266903648382923}, \
   {-982.43792032034157882, -251.393850909817774198, -48.2464593701711129338, 5.45654600348572840543, 55.5555555555555555556, 7.10799367658338150602, 1.0, 0.262074139420889660714, 0.0686828545531999120685, 0.018, -11212.4396631232758396}}
#define GWT_NODE34_LITERALS {1.42262352803113824098, 1.4814971108637783107, 1.53960071783900203869, 1.5969822136263238218, 1.65368435914272468323, 1.70974556228632557231, 1.76520049047833232268, 1.82008057513937784433, 1.87441443071783610951, 1.92822820546716415098}
#define GWT_NODEINV_LITERALS {0.625, 0.592105263157894736842, 0.5625, 0.535714285714285714286, 0.511363636363636363636, 0.489130434782608695652, 0.46875, 0.45, 0.432692307692307692308, 0.416666666666666666667}

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
  double iM, eta, ieta, delta, cM, lM, cfr, lfr, M34;  // M^(1/3), ln M, f_ref^(1/3), ln f_ref, M^(3/4)
  double xr, xd, x3, h;                     // ringdown, damping, peak in M f; half the intermediate range
  double v1, d1, v3, d3, ins1, dins1;       // connection values (derivatives by M f)
  double l2, i2, p2, rx, at2;               // at x2 = xr / 2: ln, 1/x2, x2^(3/4); xr / xd; the atan there
  double a[5];                              // intermediate amplitude in u = (M f - xm) / h
  double phi_fref;
  int have_phi, pad;
  double sn[5], cn[5];                      // of the hour angle, DEC, psi, inclination, phiRef
  double node[kPv2ShiftNodes];
};

// The divisions and the root every part needs: eta and sqrt(1 - 4 eta) rounded
// as the reference's (near equal masses the root shows the last bit of eta); 1/M, 1/eta.
GW_HDNI void fast_eta(FastX &x, const GenParams &in) {
  const double m1 = in.mass1 * kMsolSec, m2 = in.mass2 * kMsolSec, M = m1 + m2;
  x.eta = (m1 * m2) / (M * M);
  x.delta = sqrt(1. - 4 * x.eta);
}
GW_HDNI void fast_inverses(FastX &x, const GenParams &in) {
  const double m1 = in.mass1 * kMsolSec, m2 = in.mass2 * kMsolSec, M = m1 + m2;
  x.iM = 1. / M;
  x.ieta = (M * M) / (m1 * m2);
  x.M34 = sqrt(M * sqrt(M));
}
GW_HD FastCore fast_core(const GenParams &in, const FastX &x) {
  FastCore k;
  k.m1 = in.mass1 * kMsolSec;
  k.m2 = in.mass2 * kMsolSec;
  k.M = k.m1 + k.m2;
  k.iM = x.iM;
  k.eta = x.eta;
  k.ieta = x.ieta;
  k.delta = x.delta;
  k.c1 = in.spin1[2];
  k.c2 = in.spin2[2];
  k.cs = 0.5 * (k.c1 + k.c2);
  k.ca = 0.5 * (k.c1 - k.c2);
  const double chi_eff = (k.m1 * k.c1 + k.m2 * k.c2) * k.iM;
  k.chi_pn = chi_eff - ((38. / 113) * k.eta) * (2 * k.cs);
  return k;
}
GW_HD void fast_store(Source &s, const GenParams &in, const FastCore &k) {
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
  s.f1_phase = 0.018 * k.iM;
  s.f1 = 0.014 * k.iM;
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
// Inspiral amplitude and phase with their derivatives at M f = 0.014 and 0.018
// as rows of literals: rows 0, 1 (amplitude, derivative) over pn_amp[2..6],
// rho[0..2]; rows 2, 3 (phase, derivative) over pn_phase[2, 3, 4, 7, 8, 10] and,
// apart, sigma[1..4].
constexpr int kLowRows = 4, kLowPn = 6, kLowFit = 4;
#define GWT_LOW_ROWS_INIT GWT_LOW_ROWS_LITERALS
static const double gwt_low_rows_h[kLowRows][kLowPn + kLowFit + 1] = GWT_LOW_ROWS_INIT;
#if defined(__CUDACC__)
static __device__ const double gwt_low_rows_d[kLowRows][kLowPn + kLowFit + 1] = GWT_LOW_ROWS_INIT;
#endif
GW_HDNI void fast_low(const ModelD &m, FastX &x, int row) {
#if defined(__CUDA_ARCH__)
  const double *t = gwt_low_rows_d[row];
#else
  const double *t = gwt_low_rows_h[row];
#endif
  const bool amp = row < 2;
  const double *p = amp ? m.pn_amp : m.pn_phase;
  const double c[kLowPn] = {p[2], p[3], p[4], p[amp ? 5 : 7], p[amp ? 6 : 8], p[amp ? 1 : 10]};  // pn_amp[1] is zero
  const double *f = amp ? m.l.rho : m.l.sigma + 1;  // rho[3] is zero
  double s = t[kLowPn + kLowFit], n = 0.0;
#pragma unroll
  for (int j = 0; j < kLowPn; j++) s = fma(t[j], c[j], s);
#pragma unroll
  for (int j = 0; j < kLowFit; j++) n = fma(t[kLowPn + j], f[j], n);
  if (amp) {
    s += n;
    if (row == 0) x.v1 = s;
    else x.d1 = s;
  } else {
    s = fma(m.s.k_tf2, s, m.s.inv_eta * n);
    if (row == 2) x.ins1 = s - kPi / 4.;
    else x.dins1 = s;
  }
}
// Intermediate and ringdown phase terms at x2 = xr / 2.
GW_HDNI void fast_f2_powers(FastX &x) {
  const double x2 = 0.5 * x.xr;
  x.l2 = log(x2);
  x.i2 = 1. / x2;
  x.p2 = sqrt(x2 * sqrt(x2));
}
GW_HDNI void fast_f2_atan(const ModelD &m, FastX &x) {
  x.rx = x.xr / x.xd;
  x.at2 = atan((0.5 - m.l.alpha[5]) * x.rx);
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
  const double y2 = (0.5 - l.alpha[5]) * x.rx;
  const double dmr = l.alpha[2] * (i2 * i2) + l.alpha[3] * (x.p2 * i2) + l.alpha[4] / (x.xd * (1. + y2 * y2));
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
#if defined(__CUDA_ARCH__)
GW_HD double fast_rsqrt(double v) { return rsqrt(v); }
#else
GW_HD double fast_rsqrt(double v) { return 1.0 / std::sqrt(v); }
#endif
// Euler angle coefficients (pv2_euler_coeffs, IMRPhenomP.cpp:65-144): epsilon's
// and, with chi_p's terms added, alpha's.
GW_HDNI void fast_pv2_euler(ModelP &pm, const Source &s) {
  const double iq = 1. / s.q, im2 = 1. + iq, m2 = 1. / im2, m1 = m2 * iq, d = m1 - m2;
  const double n = m1 * m2, in = 1. / n, chil = s.chil, c2 = s.chip * s.chip;
  const double dn = d * im2, n2 = n * n, dn2 = dn * dn, m2s = m2 * m2, dm = d * m2, cm = chil * m2s, cd = chil * dm;
  const double c2l = chil * chil;
  double *e = pm.ec, *a = pm.ac;
  e[0] = -35. / 192 - (5. / 64) * dn;
  e[1] = -in * ((15. / 128) * cd + (35. / 128) * cm);
  e[2] = -5515. / 3072 - (4555. / 7168) * dn - n * (515. / 384 + (15. / 256) * dn2 + (175. / 256) * dn);
  e[3] = -(35. * kPi / 48) - (5. * kPi / 16) * dn + (5. / 16) * (d * d) * chil + (5. / 3) * cd + (2545. / 1152) * cm +
         in * ((2035. / 21504) * cd + (2995. / 9216) * cm);
  const double q4 = (15. / 128) * dm * m2s + (35. / 128) * (m2s * m2s);  // (15 d m2^3 + 35 m2^4) / 128
  e[4] = 4.318908476114694 + (27895885. / 2.1676032e7) * dn +
         n * (39695. / 86016 + (1615. / 28672) * dn2 - (265. / 14336) * dn) +
         n2 * (955. / 576 + (15. / 1024) * (dn2 * dn) + (35. / 256) * dn2 + (2725. / 3072) * dn) -
         (kPi * in) * ((15. / 16) * cd + (35. / 16) * cm) +
         (c2l * in) * ((375. / 256) * (dm * dm) + (1815. / 256) * (dm * m2s) + (1645. / 192) * (m2s * m2s));
  const double in2 = in * in, m4 = m2s * m2s;
  a[0] = e[0];
  a[1] = e[1];
  a[2] = e[2] - c2 * in2 * q4;
  a[3] = e[3] - c2 * chil * (in2 * in) * m4 * ((5. / 128) * dm + (35. / 384) * m2s);
  a[4] = e[4] + c2 * (in2 * (-(485. / 14336) * (dm * m2s) + (475. / 6144) * m4) +
                      in * ((15. / 256) * (dm * dm) + (145. / 512) * (dm * m2s) + (575. / 1536) * m4) +
                      (c2l - 0.25 * c2) * (in2 * in2) * m4 * q4);
}
// chi_p and the in-plane angular momenta (PhenomPv2_Param_Transform,
// IMRPhenomP.cpp:1082-1210; reduced: :822-938), before the ringdown part.
GW_HDNI void fast_pv2_spins(Source &s, const GenParams &in) {
  const double m1 = in.mass1 * kMsolSec, m2 = in.mass2 * kMsolSec, M = m1 + m2, im1 = 1. / m1;
  const double q21 = m2 * im1, c1 = in.spin1[2], c2 = in.spin2[2];
  s.chil = c1 + q21 * c2;  // (1 + q) / q chi_eff
  const double m1_2 = m1 * m1, m2_2 = m2 * m2;
  const double q = m1 / m2;
  s.q = q;
  s.phip = in.phip;
  s.chip = in.chip;
  if (!((in.chip + 1) > kCompThresh)) {
    const double S1 = m1_2 * sqrt(in.spin1[1] * in.spin1[1] + in.spin1[0] * in.spin1[0]);
    const double S2 = m2_2 * sqrt(in.spin2[1] * in.spin2[1] + in.spin2[0] * in.spin2[0]);
    const double A1 = 2 + 1.5 * q21, A2 = 2 + 1.5 * q;
    const double a1 = A1 * S1, a2 = A2 * S2;
    s.chip = (a2 > a1 ? a2 : a1) / (m2 > m1 ? A2 * m2_2 : A1 * m1_2);
  }
  const double iM2 = 1.0 / (M * M);
  s.SP = s.chip * (m1_2 * iM2);
  s.SL = (c1 * m1_2 + c2 * m2_2) * iM2;
}
// The rotation by -theta_J near the axis, in the reference's order (a function of
// its own: rarely taken, and the parts are short of instruction fetch).
GW_HDNI void fast_pv2_near_axis(const Source &s, double p2, double &sB, double &cB) {
  const double m1_2 = s.mass1 * s.mass1, m2_2 = s.mass2 * s.mass2;
  Pows pw, pp;
  precalc_powers_PI(pp);
  precalc_powers_ins(s.f_ref, s.M, pw);
  const double L0 = s.M * s.M * L2PN(s.eta, pw.MF2third, pp.PI2third), z = L0 + m1_2 * s.spin1z + m2_2 * s.spin2z;
  sincos(-acos(z / sqrt(p2 + z * z)), &sB, &cB);
}
// The J frame (IMRPhenomP.cpp:1130-1210): rotations by -phi_J about z, -theta_J
// about y and kappa about z, their sines and cosines from the components that
// define the angles.  sn/cn: of the inclination [3] and phiRef [4].
// part 0: all but alpha0; part 1: alpha0 (the same instructions up to the one atan2
// each takes, for two lanes); part 2: both.
GW_HDNI void fast_pv2_frame(Source &s, ModelP &pm, const GenParams &in, const FastX &x, int part) {
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
  const double p2 = Jx * Jx + Jy * Jy, ip = p2 > 0 ? fast_rsqrt(p2) : 0.0, iJ = fast_rsqrt(p2 + Jz * Jz);
  const double cA = p2 > 0 ? Jx * ip : 1.0, sA = -Jy * ip;
  double cB = Jz * iJ, sB = -(p2 * ip) * iJ;
  // Near the axis as the reference's theta_J = acos(J_z / J), which has few digits
  // there, makes them (with J_z's bits, in its order): alpha_0 follows sB's sign
  // alone, and J against the axis leaves theta_J = pi, whose sine is pi's rounding.
  if (p2 == 0) {
    cB = Jz < 0 ? -1.0 : 1.0;
    sB = Jz < 0 ? -1.2246467991473532e-16 : 0.0;
  } else if (p2 < 1e-10 * (Jz * Jz)) {
    fast_pv2_near_axis(s, p2, sB, cB);
  }
  const double si = x.sn[3], ci = x.cn[3], sr = x.sn[4], cr = x.cn[4];
  // N = (si cos(pi/2 - phiRef), si sin(pi/2 - phiRef), ci) through A and B
  double tx = si * sr, ty = si * cr, t1 = tx * cA - ty * sA;
  const double ny = tx * sA + ty * cA;
  const double nx = t1 * cB + ci * sB, nz = -t1 * sB + ci * cB;
  const double r2 = nx * nx + ny * ny, ir = r2 > 0 ? fast_rsqrt(r2) : 0.0, r = r2 * ir;
  const double cK = r2 > 0 ? nx * ir : 1.0, sK = -ny * ir;
  // azimuths: of J in the source frame; of L = z through A, B and K
  if (part == 2) {
    s.phi_aligned = p2 > 0 ? -atan2(Jy, Jx) : 0.0;
    s.alpha0 = atan2(sB * sK, sB * cK);
  } else {
    const double az = atan2(part ? sB * sK : Jy, part ? sB * cK : Jx);
    if (part) {
      s.alpha0 = az;
      return;
    }
    s.phi_aligned = p2 > 0 ? -az : 0.0;
  }
  // X through A, B and K
  tx = -ci * sr;
  ty = -ci * cr;
  t1 = tx * cA - ty * sA;
  const double xy = tx * sA + ty * cA, xx = t1 * cB + si * sB, xz = -t1 * sB + si * cB;
  const double px = xx * cK - xy * sK, py = xx * sK + xy * cK;
  // zeta = atan2(X . Q, X . P), P = -y, Q = (Nz, 0, -Nx): cos and sin of 2 zeta
  const double P = -py, Q = px * nz - xz * r, n2 = P * P + Q * Q, in2 = n2 > 0 ? 1.0 / n2 : 0.0;
  pm.c2z = n2 > 0 ? (P * P - Q * Q) * in2 : 1.0;
  pm.s2z = 2.0 * P * Q * in2;
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
  const double rel = 0.8 + j * (0.4 / (kPv2ShiftNodes - 1));
  const double pow34[kPv2ShiftNodes] = GWT_NODE34_LITERALS, pow1[kPv2ShiftNodes] = GWT_NODEINV_LITERALS;
  double p34 = 0.0, inv = 0.0;
#pragma unroll
  for (int q = 0; q < kPv2ShiftNodes; q++)
    if (q == j) {
      p34 = pow34[q];  // (2 rel)^(3/4)
      inv = pow1[q];   // 1 / (2 rel)
    }
  return -l.alpha[2] * (x.i2 * inv) + ((4. / 3) * l.alpha[3]) * (x.p2 * p34) +
         l.alpha[4] * atan((rel - l.alpha[5]) * x.rx);
}
// The natural spline's slope halfway between the middle ones of ten even
// nodes: sum_k w_k (y_(5+k) - y_(4-k)) / spacing (exact for linear terms).
GW_HDNI double fast_pv2_time_shift(const ModelD &m, const FastX &x) {
  const double w[5] = {1.2990196078431372549, -0.14705882352941176471, 0.039215686274509803922,
                       -0.0098039215686274509804, 0.0016339869281045751634};
  if (!m.s.shift_time || !(x.xr > 0)) return 0.0;
  double t = 0.0;
  for (int k = 0; k < 5; k++) t += w[k] * (x.node[5 + k] - x.node[4 - k]);
  const double slope = m.l.alpha[1] + t * ((kPv2ShiftNodes - 1) / 0.4) * (0.5 * x.i2);
  return -(m.s.inv_eta * m.s.M * slope) * (1.0 / (2. * kPi));
}

// ---- the grid's coefficients (mixed_phase_coeffs, mixed_amp_coeffs, mixed_regions) ----
// The inspiral series' coefficient j of n^((j - 5)/3), j = 0..11.
GW_HDNI void fast_ins_phase(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o, int j) {
  const Source &s = m.s;
  const double cu = x.cM * g.c13, iMdf = x.iM * g.idf, K = s.k_tf2 * m.pi.PIminus_5third, *pn = m.pn_phase;
  const double Lc = kLnPi + x.lM + g.ln;
  // the factor of cu^(j - 5): a constant times a coefficient, without branches
  // (lanes hold different j)
  const double *src = j < 8 ? pn + (j == 5 ? 8 : j == 6 ? 10 : j) : m.l.sigma + (j - 7);
  constexpr double kP1 = 1.4645918875615231, kP2 = kP1 * kP1;  // pi^(1/3)
  double c = j == 1 ? 0.0 : 1.0;
  c = j == 2 ? kP2 : c;
  c = j == 3 ? kPi : c;
  c = j == 4 ? kP1 * kPi : c;
  c = j == 5 ? kP2 * kPi : c;
  c = j == 6 ? kPi * kPi : c;
  c = j == 7 ? kP1 * kPi * kPi : c;
  c = j == 9 ? 0.75 : c;
  c = j == 10 ? 0.6 : c;
  c = j == 11 ? 0.5 : c;
  const double ex = j == 5 ? pn[9] : j == 6 ? -pn[11] : 0.0;
  const double q = (j < 8 ? K : s.inv_eta) * (c * (*src + ex * Lc)) - (j == 5 ? kPi / 4. : 0.0);
  // ... and the power: cu^-5 = cu / (cu^3)^2, cu^3 = M df
  const double cu2 = cu * cu, cu4 = cu2 * cu2;
  double p = (cu * iMdf) * iMdf;
  if (j & 1) p *= cu;
  if (j & 2) p *= cu2;
  if (j & 4) p *= cu4;
  if (j & 8) p *= cu4 * cu4;
  o.qi[j] = q * p;
  if (j == 5) o.bi0 = K * m.pi.PI5third * pn[9];
  if (j == 6) o.bi1 = -(K * m.pi.PIsquare) * pn[11] * cu;
}
// Intermediate and ringdown phase, after fast_connect.
GW_HDNI void fast_phase_coeffs(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o) {
  const Source &s = m.s;
  const Lambda &l = m.l;
  const double Mdf = s.M * g.df, iMdf = x.iM * g.idf, Lx = x.lM + g.ln;
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
}
// The atan's centre and width in bins.
GW_HDNI void fast_atan_coeffs(const ModelD &m, const GridConst &g, MixedReq &o) {
  const double nc = m.l.alpha[5] * m.s.fRD * g.idf, nci = floor(nc);
  o.n_c = (int)nci;
  o.ncfrac = (float)(nc - nci);
  o.inv_nw = (float)(g.df / m.s.fdamp);
}
// Inspiral amplitude coefficient j of n^(j/3), j = 0..9.
GW_HDNI void fast_ins_amp(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o, int j) {
  const double cu = x.cM * g.c13, *pa = m.pn_amp;
  const double *src = j < 7 ? pa + j : m.l.rho + (j - 7);
  constexpr double kP1 = 1.4645918875615231, kP2 = kP1 * kP1;  // pi^(1/3)
  double c = 1.0;
  c = j == 2 ? kP2 : c;
  c = j == 3 ? kPi : c;
  c = j == 4 ? kP1 * kPi : c;
  c = j == 5 ? kP2 * kPi : c;
  c = j == 6 ? kPi * kPi : c;
  const double a = c * *src;
  const double cu2 = cu * cu, cu4 = cu2 * cu2;
  double p = 1.0;
  if (j & 1) p *= cu;
  if (j & 2) p *= cu2;
  if (j & 4) p *= cu4;
  if (j & 8) p *= cu4 * cu4;
  split_f(a * p, o.ai[j], o.ai_lo[j]);
}
// Intermediate amplitude: coefficients j0, j0 + step, ... of (n - n_mid)^j.
GW_HDNI void fast_int_amp(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o, int j0, int step) {
  // u = (n - n_m) Mdf / h, n_m the middle of the range in bins
  const double nm = 0.5 * (m.s.f1 + m.s.f3) * g.idf, nmid = floor(nm);
  o.n_mid = (int)nmid;
  const double ih = 1.0 / x.h, sc = m.s.M * g.df * ih;
  double e[5];
  fast_shift_quartic(x.a, sc, (nmid - nm) * sc, e);
#pragma unroll
  for (int j = 0; j < 5; j++)
    if ((j - j0) % step == 0) split_f(e[j], o.ei[j], o.ei_lo[j]);
}
GW_HDNI void fast_ring_amp(const ModelD &m, const FastX &x, const GridConst &g, MixedReq &o) {
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
// Region start q = 0..4: f1, f1_phase, f3, f2_phase, the cut (last non-zero bin).
GW_HDNI int fast_region(const ModelD &m, const GridConst &g, MixedReq &o, int q) {
  const Source &s = m.s;
  const double *fp = q == 0 ? &s.f1 : q == 1 ? &s.f1_phase : q == 2 ? &s.f3 : q == 3 ? &s.f2_phase : &m.fcut;
  const double fb = *fp;
  const int n = fast_grid_first(fb, g, q >= 2);
  if (q == 0) o.n_f1 = n;
  if (q == 1) o.n_f1p = n;
  if (q == 2) o.n_f3 = n;
  if (q == 3) o.n_f2p = n;
  if (q == 4) o.n_cut = n - 1;
  return n;
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

// Whether the phase terms that the two-float bins carry are small enough
// (kAccMaxTurns): their largest values are at M f = 0.018, xr / 2 and the cut 0.2.
GW_HDNI int fast_range_d(const ModelD &m, const FastX &x) {
  const Lambda &l = m.l;
  const double v = fabs(l.alpha[2]) * x.i2 + (4. / 3) * kFast34 * fabs(l.alpha[3]) + fabs(l.alpha[4]);
  return v * m.s.inv_eta < kAccMaxTurns * 2 * kPi ? 0 : 1;  // 1 for NaN
}
GW_HDNI int fast_range_p(const ModelP &pm) {
  // w = pi 0.018 .. pi 0.2: w^(-1/3) at the one end, w^(1/3) at the other, |ln w| < 2.9
  constexpr double i = 1.0 / kFastV, t = kFastVc, L = 2.9;
  const double *a = pm.ac, *e = pm.ec;
  const double va = i * (fabs(a[2]) + i * (fabs(a[1]) + i * fabs(a[0]))) + L * fabs(a[3]) + t * fabs(a[4]);
  const double ve = i * (fabs(e[2]) + i * (fabs(e[1]) + i * fabs(e[0]))) + L * fabs(e[3]) + t * fabs(e[4]);
  return va < kAccMaxTurns * 2 * kPi && 2.0 * ve < kAccMaxTurns * 2 * kPi ? 0 : 1;
}
// Finalize factors of detector d: f[0..4] (mixed_det_factors_a).
GW_HDNI void fast_det_factor(const Request &r, int d, double A, double w, double ds, double *f) {
  double G1, G2;
  mixed_det_G(r, d, G1, G2);
  if (r.approximant == kPhenomPv2) {
    const double h = -0.5 * A * A * w, k = A * ds;
    f[0] = h * G1 * G1;
    f[1] = h * G2 * G2;
    f[2] = 2.0 * h * G1 * G2;
    f[3] = k * G1;
    f[4] = k * G2;
  } else {
    const double g = G1 * G1 + G2 * G2;
    f[0] = -0.5 * A * A * w * g;
    f[1] = A * ds * sqrt(g);
    f[2] = f[3] = f[4] = 0.0;
  }
}
// Entry e of the factors, the weighted |h|^2 sums folded where the detectors
// share their weights (mixed_fold_shared_weights).  An infinite factor of the
// Pv2 cross sum Re(h+ hx*), of either sign, gives way to those of |h+|^2 and
// |hx|^2: log L goes to -inf with |h|^2.
GW_HD double fast_factor_entry(const double (*f)[kAccPerDet], int e, int ndet, bool pv2, bool shared) {
  const int d = e / kAccPerDet, k = e - d * kAccPerDet;
  if (d >= ndet) return 0.0;
  double v = f[d][k];
  if (shared && k < (pv2 ? 3 : 1)) {
    if (d) return 0.0;
    for (int q = 1; q < ndet; q++) v += f[q][k];
  }
  return pv2 && k == 2 && !(fabs(f[d][0]) < 1e300) && f[d][0] == f[d][0] ? 0.0 : v;
}
GW_HD bool fast_shared(const unsigned long long *wkey, int ndet) {
  bool same = ndet > 1;
  for (int d = 1; d < ndet; d++) same = same && wkey[d] == wkey[0];
  return same;
}
// Detectors d0, d0 + step, ...: projections, phases.
#if defined(__CUDACC__)
// the detectors in global memory: lanes read different ones
static __device__ const double gwt_det_tensor_g[9][9] = GWT_DET_TENSOR_INIT;
static __device__ const double gwt_det_location_g[9][3] = GWT_DET_LOCATION_INIT;
static __device__ const double gwt_det_geometric_g[9] = GWT_DET_GEOMETRIC_INIT;
#endif
#if defined(__CUDA_ARCH__)
#define GWT_G(name) name##_g
#else
#define GWT_G(name) name##_h
#endif
GW_HDNI void fast_antenna(Request &r, const FastX &x, const int *dets, int d0, int step) {
  const double sg = x.sn[0], cg = x.cn[0], sd = x.sn[1], cd = x.cn[1], sp = x.sn[2], cp = x.cn[2];
  const double X[3] = {-cp * sg - sp * cg * sd, -cp * cg + sp * sg * sd, sp * cd};
  const double Y[3] = {sp * sg - cp * cg * sd, sp * cg + cp * sg * sd, cp * cd};
  const double e0 = cd * cg, e1 = cd * -sg, e2 = sd;
  for (int d = d0; d < r.ndet && d < kMaxDet; d += step) {
    const double *D = GWT_G(gwt_det_tensor)[dets[d]], geo = GWT_G(gwt_det_geometric)[dets[d]];
    const double *l1 = GWT_G(gwt_det_location)[dets[0]], *l2 = GWT_G(gwt_det_location)[dets[d]];
    double fp = 0.0, fc = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {  // detector_util.cpp:901-1015, 1158-1160
      const double DX = D[i * 3] * X[0] + D[i * 3 + 1] * X[1] + D[i * 3 + 2] * X[2];
      const double DY = D[i * 3] * Y[0] + D[i * 3 + 1] * Y[1] + D[i * 3 + 2] * Y[2];
      fp += X[i] * DX - Y[i] * DY;
      fc += X[i] * DY + Y[i] * DX;
    }
    r.det[d].fp = fp * geo;
    r.det[d].fc = fc * geo;
    // detector_util.cpp:760-780
    r.det[d].tau = ((l1[0] - l2[0]) * e0 + (l1[1] - l2[1]) * e1 + (l1[2] - l2[2]) * e2) * (-2 * kPi / kC);
  }
}
GW_HDNI void fast_det_phase(const Request &r, double df, MixedReq &o, int d0, int step) {
  mixed_det_phase(r, df, o, d0, step);
}
GW_HDNI void fast_det_phase(const Request &r, double df, AccReq &o, int d0, int step) {
  acc_det_phase(r, df, o, d0, step);
}

// The parts in order (host): request_prologue, and the FP64 form's constants.
inline int fast_request(Request &r, FastX &x, const GenParams &in, int approximant, const int *dets, int ndet,
                        const double *qnm) {
  r.approximant = approximant;
  r.ndet = ndet;
  const bool pv2 = approximant == kPhenomPv2;
  ModelD &m = r.m;
  fast_eta(x, in);
  fast_inverses(x, in);
  const FastCore k = fast_core(in, x);
  m.s.pv2 = pv2;
  fast_store(m.s, in, k);
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
  fast_amp0(m, x, in, k);
  if (pv2) fast_pv2_spins(m.s, in);
  fast_ring(m.s, x, k, qnm);
  fast_high(m, x);
  for (int i = 0; i < kLowRows; i++) fast_low(m, x, i);
  fast_f2_powers(x);
  fast_f2_atan(m, x);
  fast_fref_phase(m, x);
  if (pv2) {
    fast_pv2_frame(m.s, r.p, in, x, 2);
    fast_pv2_euler(r.p, m.s);
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
                    const double *wscale, const unsigned long long *wkey) {
  const bool pv2 = r.approximant == kPhenomPv2;
  o.m.approximant = r.approximant;
  o.m.status = r.m.status;
  o.m.ndet = r.ndet;
  for (int q = 0; q < 5; q++) fast_region(r.m, g, o.m, q);
  for (int j = 0; j < 12; j++) fast_ins_phase(r.m, x, g, o.m, j);
  fast_phase_coeffs(r.m, x, g, o.m);
  fast_atan_coeffs(r.m, g, o.m);
  for (int j = 0; j < 10; j++) fast_ins_amp(r.m, x, g, o.m, j);
  fast_int_amp(r.m, x, g, o.m, 0, 1);
  fast_ring_amp(r.m, x, g, o.m);
  if (pv2) fast_pv2_coeffs(r, x, g, o.m);
  o.m.A_scale = fast_a_scale(r, g);
  double f[kMaxDet][kAccPerDet];
  for (int d = 0; d < r.ndet; d++) fast_det_factor(r, d, o.m.A_scale, wscale[d], dscale[d], f[d]);
  o.m.wshared = fast_shared(wkey, r.ndet) ? 1 : 0;
  for (int e = 0; e < kMaxDet * kAccPerDet; e++) o.m.fc[e] = fast_factor_entry(f, e, r.ndet, pv2, o.m.wshared != 0);
  fast_det_phase(r, g.df, o, 0, 1);
  acc_phase_coeffs(r, g.df, o);
  acc_amp_coeffs(r, g.df, o);
  if (pv2) acc_pv2_coeffs(r, g.df, o);
  o.fp64_phase = fast_range_d(r.m, x) | (pv2 ? fast_range_p(r.p) : 0);
  return o.m.status;
}

}  // namespace gwt

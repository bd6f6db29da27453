// acc_check.cpp -- TEST BUILD ONLY: the two-float arithmetic, the bins of the
// FP64 form built on it and the batched prologue (two_float.h, phenom_acc.h,
// phenom_fast.h) compiled for the host.
// Compiled with -ffp-contract=off: the error-free sums need every operation
// rounded by itself.
#include <cmath>
#include <vector>

#include "../../gw_analysis_tools_gb300/csrc/phenom_fast.h"

using namespace gwt;

static std::vector<double> g_qnm;
static const double *qnm() {
  if (g_qnm.empty()) {
    g_qnm.resize(kQnmArrays * kQnmLen);
    qnm_fill(g_qnm.data(), gwt_qnm_a_h, gwt_qnm_fring_h, gwt_qnm_fdamp_h);
  }
  return g_qnm.data();
}
static AccLut g_lut;
static const AccLut &lut() {
  static bool done = false;
  if (!done) ff_fill_tables(g_lut.turn, g_lut.ex);
  done = true;
  return g_lut;
}

template <int NDET>
static void bins(const AccReq &x, int n0, int N, const AccTables &tb, const std::vector<std::vector<ff4>> &wd,
                 const std::vector<std::vector<ff>> &w, const std::vector<float> &dev, double *sums) {
  const bool pv2 = x.m.approximant == kPhenomPv2;
  const int na = pv2 ? kAccPerDet : 2;
  for (int k0 = 0; k0 < N; k0 += 32) {  // a kernel thread sums a few tens of bins
    ff acc[NDET * kAccPerDet] = {};
    for (int k = k0; k < N && k < k0 + 32; k++) {
      const int n = n0 + k;
      if (n > x.m.n_cut) break;
      ff4 a[NDET];
      ff b[NDET];
      for (int d = 0; d < NDET; d++) {
        a[d] = wd[d][k];
        b[d] = w[d][k];
      }
      const AccBin bin{n, acc_dev_turns(x, dev[k])};
      if (pv2) acc_bin_p<NDET>(x, bin, tb, lut(), a, b, false, acc);
      else acc_bin_d<NDET>(x, bin, tb, lut(), a, b, false, acc);
    }
    for (int d = 0; d < NDET; d++)
      for (int j = 0; j < na; j++) sums[d * kAccPerDet + j] += ff_value(acc[d * na + j]);
  }
}

extern "C" {

// Worst errors over n random arguments: cos/sin of turns, exp, atan, turns, division, 1/sqrt.
void gwa_worst(unsigned long long seed, int n, double *out) {
  for (int i = 0; i < 6; i++) out[i] = 0;
  unsigned long long g = seed;
  auto rnd = [&]() {
    g ^= g << 13;
    g ^= g >> 7;
    g ^= g << 17;
    return g;
  };
  const long double two_pi = 6.283185307179586476925286766559L, q64 = 18446744073709551616.0L;
  auto up = [&](int i, long double e) { out[i] = std::fmax(out[i], (double)fabsl(e)); };
  for (int it = 0; it < n; it++) {
    unsigned long long q = rnd();
    if (it % 5 == 0) q >>= it % 60;                                     // near zero
    if (it % 7 == 0) q = (q & 3ull) << 62 | (q >> (20 + it % 40));      // near the quarter turns
    ff c, s;
    ff_turns_sincos(q, lut().turn, c, s);
    const long double th = (long double)q / q64 * two_pi;
    up(0, cosl(th) - ((long double)c.h + c.l));
    up(0, sinl(th) - ((long double)s.h + s.l));
    const double u = (double)(rnd() >> 11) * 0x1p-53;
    const ff z = ff_split(8.0 * u - 6.0), e = ff_exp(z, lut().ex);
    up(1, ((long double)e.h + e.l) / expl((long double)z.h + z.l) - 1);
    const ff y = ff_split(std::tan((u - 0.5) * 3.1415) * (it % 3 ? 1.0 : 0.01));
    ff d;
    const int i = ff_atan(y, lut().turn, d);
    up(2, (long double)i / kTurnTab * two_pi + d.h + d.l - atanl((long double)y.h + y.l));
    const ff t = ff_split((u - 0.5) * 40);
    long double fr = (long double)t.h + t.l - (long double)ff_turns_q64(t) / q64;
    up(3, fr - rintl(fr));
    const ff a = ff_split(u + 0.1), v = ff_div(y, a), w = ff_rsqrt(a);
    up(4, ((long double)v.h + v.l) * ((long double)a.h + a.l) / ((long double)y.h + y.l) - 1);
    up(5, ((long double)w.h + w.l) * sqrtl((long double)a.h + a.l) - 1);
  }
}

// log L of one request on the grid f_k ~ (n0 + k) df.  mode bit 0: the FP64
// phase series at every bin; bit 1: the prologue of phenom_fast.h.
double gwa_loglik(const GenParams *pin, int approx, double T_segment, int n0, const double *f, int N, int ndet,
                  const int *dets, const double *const *data, const double *const *psd, int mode, int *fp64_phase) {
  GenParams p = *pin;
  p.tc = T_segment - p.tc;
  const double df = (f[N - 1] - f[0]) / (N - 1);
  std::vector<float> dev(N);
  for (int k = 0; k < N; k++) dev[k] = (float)std::fma(-(double)(n0 + k), df, f[k]);
  Request r;
  FastX fx;
  if (mode & 2 ? fast_request(r, fx, p, approx, dets, ndet, qnm()) : request_prologue(r, p, approx, dets, ndet, qnm()))
    return NAN;
  std::vector<std::vector<ff4>> wd(ndet);
  std::vector<std::vector<ff>> w(ndet);
  double ds[kMaxDet], ws[kMaxDet];
  for (int d = 0; d < ndet; d++) {
    double wm = 0, dm = 0;
    std::vector<double> W(N);
    for (int k = 0; k < N; k++) {
      W[k] = (4. * (f[N / 2] - f[N / 2 - 1]) / 3.) * simpson_weight(k, N) / psd[d][k];
      wm = std::fmax(wm, W[k]);
      dm = std::fmax(dm, std::fabs(W[k] * data[d][2 * k]) + std::fabs(W[k] * data[d][2 * k + 1]));
    }
    ds[d] = dm;
    ws[d] = wm;
    for (int k = 0; k < N; k++) {
      const ff a = ff_split(W[k] * data[d][2 * k] / dm), b = ff_split(W[k] * data[d][2 * k + 1] / dm);
      wd[d].push_back(ff4{a.h, a.l, b.h, b.l});
      w[d].push_back(ff_split(W[k] / wm));
    }
  }
  AccReq x;
  const unsigned long long wk[kMaxDet] = {1, 2, 3, 4};  // no shared weights
  if (mode & 2) fast_acc(r, fx, grid_const(df), x, ds, ws, wk);
  else acc_prologue(r, df, x, ds, ws);
  if (mode & 1) x.fp64_phase = 1;
  if (fp64_phase) *fp64_phase = x.fp64_phase;
  std::vector<double> t13(n0 + N), tm53(n0 + N), tln(n0 + N), t34(n0 + N);
  std::vector<ff4> pw(n0 + N), ph(n0 + N), pv(n0 + N);
  for (int n = n0; n < n0 + N; n++) {
    t13[n] = std::cbrt((double)n);
    tm53[n] = std::pow((double)n, -5. / 3.);
    tln[n] = std::log((double)n);
    t34[n] = std::pow((double)n, 0.75);
    auto two = [](double a, double b) {
      const ff u = ff_split(a), v = ff_split(b);
      return ff4{u.h, u.l, v.h, v.l};
    };
    pw[n] = two(t13[n], std::pow((double)n, -7. / 6.));
    ph[n] = two(1.0 / n, t34[n]);
    pv[n] = two(1.0 / t13[n], tln[n]);
  }
  const AccTables tb{pw.data(), ph.data(), pv.data(), t13.data(), tm53.data(), tln.data(), t34.data(), n0 + N - 1};
  double sums[kMaxDet * kAccPerDet] = {};
  if (ndet == 1) bins<1>(x, n0, N, tb, wd, w, dev, sums);
  else if (ndet == 2) bins<2>(x, n0, N, tb, wd, w, dev, sums);
  else bins<3>(x, n0, N, tb, wd, w, dev, sums);
  return mixed_finalize(x.m, sums);
}
}

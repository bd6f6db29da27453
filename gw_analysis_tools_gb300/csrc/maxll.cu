// maxll.cu -- the likelihood maximised over arrival time and phase,
// maximized_Log_Likelihood_aligned_spin_internal (mcmc_gw.cpp:595-658) and
// maximized_Log_Likelihood_unaligned_spin_internal (:660-800), and the
// sampler's intrinsic mode that sums them over detectors
// (MCMC_likelihood_wrapper, mcmc_gw.cpp:2611-2720).
//
// Per (request, detector): HH = 4 S(|r|^2 / S_n) by Simpson's rule,
// g_k = 4 conj(d_k) r_k / S_n,k, G = DFT_N(g), and
// log L = 1/2 max_j |G_j|^2 df^2 / HH (the unaligned form: 1/4 max of lambda,
// built from the transforms of the h+ and hx products).
//
// Grid lengths N with a prime factor above 7 (32128 = 2^7 * 251 is typical)
// use Bluestein's identity nk = (n^2 + k^2 - (k - n)^2) / 2 with power-of-two
// transforms of length M >= 2N - 1:
//   G_k = e^{-i pi k^2/N} sum_n [g_n e^{-i pi n^2/N}] e^{i pi (k-n)^2/N},
// a cyclic convolution of a_n = g_n e^{-i pi n^2/N} with b_m = e^{i pi m^2/N}
// (FFT_M, a pointwise product with the transform of b, inverse FFT_M).  The
// outer factor e^{-i pi k^2/N} is never applied: every quantity taken from G
// (|G_k|^2, Re(G+_k conj(Gx_k))) is invariant to a phase common to the pair.
// The chirp phases use n^2 mod 2N in integers.
//
// GB300's FP64 rate makes FP64 transforms the bottleneck, so by default the
// transforms run in FP32 and only locate the maximum: with E a bound on the
// FP32 error of each G_k (tau * ||C||_2, from the transform's norm growth),
// every k whose FP32 value could still be the maximum (|C_k| + E >= max_j
// |C_j| - E, or the same with the lambda bound of the unaligned form) is a
// candidate, and G is evaluated exactly in FP64 at the candidates only (a
// direct sum with exactly reduced twiddles).  The result is the maximum over
// the FP64 values, i.e. the reference's maximum.  A pair with more than
// kCand candidates (a flat spectrum) sends the batch to the FP64 transforms
// (also selected by GWGPU_MAXLL=fp64).
//
// On uniform grids the waveform, the products g and the refinement's sums run on
// pairs of FP32 numbers (phenom_acc.h): as FP64 they were 70 % of the time.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/gwgpu.h"
#include "capi_internal.h"
#include "conv.h"
#include "cufft_rt.h"
#include "kernels.h"

namespace {

using gwk::StreamDev;
using gwt::Request;

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;

// e^{sign i pi m^2 / N}, the phase reduced exactly (m^2 mod 2N in integers).
__device__ __forceinline__ double2 chirp(long long m, int N, double sign) {
  const long long t = (m * m) % (2LL * N);
  double sn, cs;
  sincospi((double)t / (double)N, &sn, &cs);
  return make_double2(cs, sign * sn);
}

// ------------------------------------------------------------------ kernels
// Block (x, r): bins x*256.. of request r, for each of its detectors d (pair
// q = r*ndet + d); rows of g have stride ld (N, or M for Bluestein, the bins
// N..M-1 zero).  The waveform is evaluated once per bin and request, on the
// grid of the request's first detector (the reference evaluates it once on
// local_freqs[0], mcmc_gw.cpp:2651-2653, 2697-2701).
//
// Aligned (UN = false): g = 4 conj(d) h / S into row q, and the block partial
// sums of w_k |h|^2 / S (Simpson weights w).  h is the model's h+ (the
// horizon frame at theta = phi = psi = 0 and inclination 0 that the sampler's
// intrinsic mode uses gives F+ = 1, Fx = 0), or a given response per pair.
// Unaligned (UN = true): the same for h+ and hx into rows 2q and 2q+1, and
// partial sums of |h+|^2/S, |hx|^2/S and Re(h+ conj(hx))/S.  The
// normalisation by sqrt(<h+|h+>) and sqrt(<hx|hx>) is applied after the
// transform (it is linear).  With Bluestein, g is multiplied by
// e^{-i pi k^2/N}.
template <bool UN>
__global__ void k_maxll_prep(const Request *__restrict__ req, const double2 *__restrict__ resp_p,
                             const double2 *__restrict__ resp_c, int ndet, const StreamDev *__restrict__ streams,
                             const int *__restrict__ handles, int N, int ld, int blue, double2 *__restrict__ g,
                             double *__restrict__ part) {
  constexpr int NS = UN ? 3 : 1, NP = UN ? 2 : 1;
  __shared__ double s_red[NS][kWarps];
  const int r = blockIdx.y;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  // a request outside the model domain contributes zeros (its result is NaN)
  double2 hp = make_double2(0.0, 0.0), hc = make_double2(0.0, 0.0);
  if (req && k < N && !req[r].m.status) {
    gwt::cd p, c;
    gwt::wave_bin(req[r], streams[handles[(size_t)r * ndet]].freqs[k], p, c);
    hp = make_double2(p.re, p.im);
    hc = make_double2(c.re, c.im);
  }
  const double2 ch = (blue && k < N) ? chirp(k, N, -1.0) : make_double2(1.0, 0.0);
  for (int dd = 0; dd < ndet; dd++) {
    const int q = r * ndet + dd;
    const StreamDev &st = streams[handles[q]];
    double acc[NS];
#pragma unroll
    for (int j = 0; j < NS; j++) acc[j] = 0.0;
    if (k < N) {
      if (!req) {
        hp = resp_p[(size_t)q * N + k];
        if (UN) hc = resp_c[(size_t)q * N + k];
      }
      const double2 d = ((const double2 *)st.data)[k];
      const double iS = st.ipsd ? st.ipsd[k] : 1.0 / st.psd[k], w = gwt::simpson_weight(k, N), s4 = 4.0 * iS;
      // 4 conj(d) h / S, then the Bluestein chirp
      double2 v = make_double2(s4 * (d.x * hp.x + d.y * hp.y), s4 * (d.x * hp.y - d.y * hp.x));
      g[((size_t)q * NP) * ld + k] = make_double2(v.x * ch.x - v.y * ch.y, v.x * ch.y + v.y * ch.x);
      acc[0] = w * ((hp.x * hp.x + hp.y * hp.y) * iS);
      if (UN) {
        v = make_double2(s4 * (d.x * hc.x + d.y * hc.y), s4 * (d.x * hc.y - d.y * hc.x));
        g[((size_t)q * NP + 1) * ld + k] = make_double2(v.x * ch.x - v.y * ch.y, v.x * ch.y + v.y * ch.x);
        acc[1] = w * ((hc.x * hc.x + hc.y * hc.y) * iS);
        acc[2] = w * ((hp.x * hc.x + hp.y * hc.y) * iS);
      }
    } else if (k < ld) {
      g[((size_t)q * NP) * ld + k] = make_double2(0.0, 0.0);
      if (UN) g[((size_t)q * NP + 1) * ld + k] = make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < NS; j++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    __syncthreads();  // the previous detector's partials have been read
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int j = 0; j < NS; j++) s_red[j][threadIdx.x >> 5] = acc[j];
    __syncthreads();
    if (threadIdx.x < NS) {
      double t = 0.0;
      for (int w = 0; w < kWarps; w++) t += s_red[threadIdx.x][w];
      part[((size_t)q * NS + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// The Bluestein kernel: B = FFT_M(b) / M is made from b_m = e^{i pi m^2/N} at
// index m (0 <= m < N) and M - m (0 < m < N), zero elsewhere.
__global__ void k_chirp_fill(double2 *__restrict__ b, int N, int M) {
  const double inv = 1.0 / (double)M;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    long long m = -1;
    if (i < N) m = i;
    else if (i > M - N) m = M - i;
    double2 v = make_double2(0.0, 0.0);
    if (m >= 0) {
      v = chirp(m, N, 1.0);
      v.x *= inv;
      v.y *= inv;
    }
    b[i] = v;
  }
}

// g[row][i] *= B[i] over all rows (the convolution's pointwise product).
__global__ void k_chirp_mul(double2 *__restrict__ g, const double2 *__restrict__ B, int M, long long total) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const double2 a = g[i], c = B[i % M];
    g[i] = make_double2(a.x * c.x - a.y * c.y, a.x * c.y + a.y * c.x);
  }
}

// Sum of v over the block (every thread gets it; s_tmp: one double per warp).
__device__ double block_sum(double v, double *s_tmp) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s_tmp[w];
  return t;
}

// One block per pair: the Simpson sums from the partials, then the maximum
// over the transform (rows of stride ld, the first N entries) and log L of the
// pair; the last block of each request sums its detectors in order.
//   aligned   (mcmc_gw.cpp:595-658): 1/2 max|G|^2 df^2 / <h|h>
//   unaligned (mcmc_gw.cpp:660-800): 1/4 max lambda, with
//     rho+ = df G+ / sqrt(<h+|h+>), rhox = df Gx / sqrt(<hx|hx>),
//     gamma = Re(rho+ conj(rhox)), I = <h+|hx> / sqrt(<h+|h+><hx|hx>),
//     lambda = (|rho+|^2 + |rhox|^2 - 2 gamma I + sqrt((|rho+|^2 - |rhox|^2)^2
//              + 4 (I |rho+|^2 - gamma)(I |rhox|^2 - gamma))) / (1 - I^2).
template <bool UN>
__global__ void k_maxll_reduce(const double2 *__restrict__ G, const double *__restrict__ part, int nblk, int N,
                               int ld, int ndet, const StreamDev *__restrict__ streams,
                               const int *__restrict__ handles, const int *__restrict__ req_status,
                               double *__restrict__ ll_pair, unsigned *__restrict__ done, double *__restrict__ out,
                               int *__restrict__ status) {
  constexpr int NS = UN ? 3 : 1, NP = UN ? 2 : 1;
  __shared__ double s_tmp[kWarps];
  __shared__ bool s_last;
  const int q = blockIdx.x, r = q / ndet;
  const StreamDev &st = streams[handles[q]];
  const double df = st.freqs[1] - st.freqs[0];  // mcmc_gw.cpp:604, also the Simpson step
  double sums[NS];
#pragma unroll
  for (int j = 0; j < NS; j++) {
    double t = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) t += part[((size_t)q * NS + j) * nblk + b];
    sums[j] = 4.0 * block_sum(t, s_tmp) * df / 3.0;
  }
  double m = 0.0;
  if (!UN) {
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
      const double2 v = G[(size_t)q * ld + k];
      m = fmax(m, v.x * v.x + v.y * v.y);
    }
  } else {
    const double ap = df / sqrt(sums[0]), ac = df / sqrt(sums[1]);
    const double I = sums[2] / (sqrt(sums[0]) * sqrt(sums[1]));
    m = -HUGE_VAL;
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
      const double2 a = G[((size_t)q * NP) * ld + k], c = G[((size_t)q * NP + 1) * ld + k];
      const double rpx = ap * a.x, rpy = ap * a.y, rcx = ac * c.x, rcy = ac * c.y;
      const double p2 = rpx * rpx + rpy * rpy, c2 = rcx * rcx + rcy * rcy;
      const double gam = rpx * rcx + rpy * rcy;
      const double lam =
          (p2 + c2 - 2 * gam * I + sqrt((p2 - c2) * (p2 - c2) + 4. * (I * p2 - gam) * (I * c2 - gam))) / (1. - I * I);
      m = fmax(m, lam);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double mx = s_tmp[0];
    for (int w = 1; w < kWarps; w++) mx = fmax(mx, s_tmp[w]);
    ll_pair[q] = UN ? 0.25 * mx : 0.5 * (mx * df * df) / sums[0];
    __threadfence();
    s_last = atomicAdd(done + r, 1u) == (unsigned)ndet - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    double ll = 0.0;
    for (int d = 0; d < ndet; d++) ll += __ldcg(ll_pair + (size_t)r * ndet + d);
    const int rs = req_status ? req_status[r] : 0;
    out[r] = rs ? __longlong_as_double(0x7ff8000000000000ll) : ll;
    if (status) status[r] = rs;
  }
}

// ======================================================= FP32 search path
constexpr int kCand = 32;              // candidates per pair
// FP32 transform error / (||a||_2 * kscale), for each entry and so for the norm.  The
// library's transforms: with a 4x margin.  conv.cu, by its operations in units of
// 2^-24: 7 for a butterfly of 16, 3 for a twiddle, so 21 for a length of 512; four
// of those, the two steps between them and the spectrum 94 at the longest rows, the
// chirp and its product 10: 6.3e-6, a margin of six.
constexpr double kTau = 4e-5;
constexpr int kMaxTwiddleRows = 12288; // shared twiddle table of the refinement: N <= 256 * this

// e^{-i pi m^2 / N} in FP32 (phase reduced exactly in integers).
__device__ __forceinline__ float2 chirp32(long long m, int N) {
  const long long t = (m * m) % (2LL * N);
  float sn, cs;
  sincospif((float)t / (float)N, &sn, &cs);
  return make_float2(cs, -sn);
}

// As k_maxll_prep, writing the exact products g (FP64, rows of N) for the
// refinement and their FP32 (chirped) copy a (rows of ld) for the search, with
// the partial sums of |g|^2 per row beside the Simpson sums:
//   aligned:   [<h|h>, |g|^2]
//   unaligned: [<h+|h+>, <hx|hx>, <h+|hx>, |g+|^2, |gx|^2]
template <bool UN>
__global__ void k_mx_prep(const Request *__restrict__ req, const double2 *__restrict__ resp_p,
                          const double2 *__restrict__ resp_c, int ndet, const StreamDev *__restrict__ streams,
                          const int *__restrict__ handles, int N, int ld, int blue, double2 *__restrict__ g64,
                          float2 *__restrict__ a32, double *__restrict__ part) {
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1;
  __shared__ double s_red[NS][kWarps];
  const int r = blockIdx.y;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double2 hp = make_double2(0.0, 0.0), hc = make_double2(0.0, 0.0);
  if (req && k < N && !req[r].m.status) {
    gwt::cd p, c;
    gwt::wave_bin(req[r], streams[handles[(size_t)r * ndet]].freqs[k], p, c);
    hp = make_double2(p.re, p.im);
    hc = make_double2(c.re, c.im);
  }
  const float2 ch = (blue && k < N) ? chirp32(k, N) : make_float2(1.f, 0.f);
  for (int dd = 0; dd < ndet; dd++) {
    const int q = r * ndet + dd;
    const StreamDev &st = streams[handles[q]];
    double acc[NS];
#pragma unroll
    for (int j = 0; j < NS; j++) acc[j] = 0.0;
    if (k < N) {
      if (!req) {
        hp = resp_p[(size_t)q * N + k];
        if (UN) hc = resp_c[(size_t)q * N + k];
      }
      const double2 d = ((const double2 *)st.data)[k];
      const double iS = st.ipsd ? st.ipsd[k] : 1.0 / st.psd[k], w = gwt::simpson_weight(k, N), s4 = 4.0 * iS;
      const double2 v = make_double2(s4 * (d.x * hp.x + d.y * hp.y), s4 * (d.x * hp.y - d.y * hp.x));
      g64[((size_t)q * NP) * N + k] = v;
      const float vx = (float)v.x, vy = (float)v.y;
      a32[((size_t)q * NP) * ld + k] = make_float2(vx * ch.x - vy * ch.y, vx * ch.y + vy * ch.x);
      acc[0] = w * ((hp.x * hp.x + hp.y * hp.y) * iS);
      if (UN) {
        const double2 u = make_double2(s4 * (d.x * hc.x + d.y * hc.y), s4 * (d.x * hc.y - d.y * hc.x));
        g64[((size_t)q * NP + 1) * N + k] = u;
        const float ux = (float)u.x, uy = (float)u.y;
        a32[((size_t)q * NP + 1) * ld + k] = make_float2(ux * ch.x - uy * ch.y, ux * ch.y + uy * ch.x);
        acc[1] = w * ((hc.x * hc.x + hc.y * hc.y) * iS);
        acc[2] = w * ((hp.x * hc.x + hp.y * hc.y) * iS);
        acc[3] = v.x * v.x + v.y * v.y;
        acc[4] = u.x * u.x + u.y * u.y;
      } else {
        acc[NS - 1] = v.x * v.x + v.y * v.y;
      }
    } else if (k < ld) {
      a32[((size_t)q * NP) * ld + k] = make_float2(0.f, 0.f);
      if (UN) a32[((size_t)q * NP + 1) * ld + k] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < NS; j++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int j = 0; j < NS; j++) s_red[j][threadIdx.x >> 5] = acc[j];
    __syncthreads();
    if (threadIdx.x < NS) {
      double t = 0.0;
      for (int w = 0; w < kWarps; w++) t += s_red[threadIdx.x][w];
      part[((size_t)q * NS + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// k_mx_prep for the intrinsic mode on uniform grids: the waveform and the products
// in two floats (g as pairs), a tile of kPrepTile bins per block; a32's rows are
// padded with zeros up to pad.
// Bound by memory: per pair and bin 16 B of data read and 16 + 8 B written (for a
// library transform the padding of a Bluestein row another 8 B per entry).  128 IMRPhenomD requests on
// 3 x 32,128 bins: 1,480 -> 97 us against the FP64 bins at
// four blocks an SM (three: 103; Pv2, 48 requests on 3 x 15,680, two: 57, one: 81); bins beyond a
// request's cut only write their zeros (242 -> 131 us), the padding none.
constexpr int kPrepTile = 2048;
// Bins of the grid below the model's cut (0 for a request outside its domain).
__device__ __forceinline__ int live_bins(const gwt::AccReq &x, int n0, int N) {
  return x.m.status ? 0 : max(0, min(N, x.m.n_cut - n0 + 1));
}
template <bool UN>
__global__ void __launch_bounds__(kBlock, UN ? 2 : 4) k_mx_prep_ff(const gwt::AccReq *__restrict__ areq, int ndet,
                                                       const StreamDev *__restrict__ streams,
                                                       const int *__restrict__ handles, const gwt::AccTables tb,
                                                       const gwt::AccLut *__restrict__ glut, int N, int ld, int pad,
                                                       int blue, const float2 *__restrict__ chirp_tab,
                                                       gwt::ff4 *__restrict__ g,
                                                       float2 *__restrict__ a32, double *__restrict__ part) {
  using namespace gwt;
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1;
  __shared__ AccLut lut;
  __shared__ __align__(16) unsigned char s_req[sizeof(AccReq)];
  __shared__ StreamDev s_st[kMaxDet];
  __shared__ ff s_sc[kMaxDet];
  __shared__ float s_un[kMaxDet];  // about 1 / s_sc, a power of two: |g|^2 is summed without its scale's square
  __shared__ double s_hs[kMaxDet], s_gs[kMaxDet], s_red[kMaxDet * NS][kWarps];
  const int r = blockIdx.y, tid = threadIdx.x;
  const AccReq &x = *(const AccReq *)s_req;
  const int k0 = blockIdx.x * kPrepTile, k1 = min(k0 + kPrepTile, pad);
  if (tid < ndet) s_st[tid] = streams[handles[(size_t)r * ndet + tid]];
  __syncthreads();
  // bins below the model's cut; g is neither written nor read beyond them
  const int n0 = s_st[0].n0, kcut = live_bins(areq[r], n0, N);
  if (k0 < kcut) {
    for (int w = tid; w < (int)(sizeof(AccLut) / 4); w += kBlock) ((unsigned *)&lut)[w] = ((const unsigned *)glut)[w];
    for (int w = tid; w < (int)(sizeof(AccReq) / 4); w += kBlock)
      ((unsigned *)s_req)[w] = ((const unsigned *)(areq + r))[w];
  }
  if (tid < ndet) {  // the streams' pairs are W d / dscale and W / wscale, W = (4 df_s / 3) s_k / S_k
    const StreamDev &st = s_st[tid];
    const double A = areq[r].m.A_scale;
    s_sc[tid] = ff_split(A * (3.0 * st.dscale / st.simpson_df));
    const int e = min(126, max(-126, s_sc[tid].h != 0.0f ? ilogbf(s_sc[tid].h) : 0));
    s_un[tid] = ldexpf(1.0f, -e);
    s_gs[tid] = ldexp(1.0, 2 * e);
    s_hs[tid] = A * A * st.wscale * (3.0 / (4.0 * st.simpson_df));
  }
  __syncthreads();
  const float *dev = s_st[0].dev;
  ff acc[kMaxDet * NS];
#pragma unroll
  for (int j = 0; j < kMaxDet * NS; j++) acc[j] = ff{0.f, 0.f};
  for (int k = k0 + tid; k < k1; k += kBlock) {
    if (k >= kcut) {
      for (int q = r * ndet * NP; q < (r + 1) * ndet * NP; q++) a32[(size_t)q * ld + k] = make_float2(0.f, 0.f);
      continue;
    }
    ff pr, pi, cr, ci;
    const uint64_t qd = dev ? acc_dev_turns(x, __ldg(dev + k)) : 0;
    acc_wave<UN>(x, n0 + k, qd, tb, lut, pr, pi, cr, ci);
    const float2 ch = blue ? __ldg(chirp_tab + k) : make_float2(1.f, 0.f);
    const float is = k == 0 || k == N - 1 ? 1.0f : (k & 1) ? 0.25f : 0.5f;  // 1 / s_k
    const ff hh = ff_norm(ff_add(ff_sqr(pr), ff_sqr(pi)));
    ff cc, hc;
    if constexpr (UN) {
      cc = ff_norm(ff_add(ff_sqr(cr), ff_sqr(ci)));
      hc = ff_norm(ff_add(ff_mul(pr, cr), ff_mul(pi, ci)));
    }
#pragma unroll
    for (int dd = 0; dd < kMaxDet; dd++) {
      if (dd >= ndet) break;
      const size_t q = (size_t)(r * ndet + dd) * NP;
      const ff4 w = acc_ld(s_st[dd].wd + k);
      const float2 wv = __ldg((const float2 *)s_st[dd].wf + k);
      const ff wk{wv.x, wv.y}, sc{s_sc[dd].h * is, s_sc[dd].l * is};
      const ff dr = ff_norm(ff_mul(ff{w.ch, w.cl}, sc)), di = ff_norm(ff_mul(ff{w.sh, w.sl}, sc));
      const float un = s_un[dd];
      auto product = [&](ff hr, ff hi, size_t row, ff &nn) {  // 4 conj(d) h / S
        const ff vr = ff_norm(ff_add(ff_mul(dr, hr), ff_mul(di, hi))), vi = ff_norm(ff_sub(ff_mul(dr, hi), ff_mul(di, hr)));
        g[row * N + k] = ff4{vr.h, vr.l, vi.h, vi.l};
        a32[row * ld + k] = make_float2(vr.h * ch.x - vi.h * ch.y, vr.h * ch.y + vi.h * ch.x);
        const float ur = vr.h * un, ui = vi.h * un;
        nn.h = fmaf(ur, ur, fmaf(ui, ui, nn.h));  // |g|^2 for the search's error bound
      };
      ff_acc(acc[dd * NS], ff_mul(wk, hh));
      if constexpr (UN) {
        ff_acc(acc[dd * NS + 1], ff_mul(wk, cc));
        ff_acc(acc[dd * NS + 2], ff_mul(wk, hc));
        product(pr, pi, q, acc[dd * NS + 3]);
        product(cr, ci, q + 1, acc[dd * NS + 4]);
      } else {
        product(pr, pi, q, acc[dd * NS + 1]);
      }
    }
  }
#pragma unroll
  for (int dd = 0; dd < kMaxDet; dd++) {
    if (dd >= ndet) break;
#pragma unroll
    for (int j = 0; j < NS; j++) {
      ff v = acc[dd * NS + j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        v = ff_add(v, ff{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)});
      if ((tid & 31) == 0) s_red[dd * NS + j][tid >> 5] = ff_value(v);
    }
  }
  __syncthreads();
  if (tid < ndet * NS) {
    double t = 0.0;
    for (int w = 0; w < kWarps; w++) t += s_red[tid][w];
    const int j = tid % NS;
    part[((size_t)r * ndet * NS + tid) * gridDim.x + blockIdx.x] = t * (j < (UN ? 3 : 1) ? s_hs : s_gs)[tid / NS];
  }
}

// The Bluestein chirp e^{-i pi k^2/N}, k < N, in FP32.
__global__ void k_chirp_tab(float2 *__restrict__ t, int N) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) t[k] = chirp32(k, N);
}

__global__ void k_chirp_mul32(float2 *__restrict__ a, const float2 *__restrict__ B, int M, long long total) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const float2 x = a[i], c = B[i % M];
    a[i] = make_float2(x.x * c.x - x.y * c.y, x.x * c.y + x.y * c.x);
  }
}

// Block max of v (every thread gets it).
__device__ float block_max(float v, float *s_tmp) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = s_tmp[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); w++) t = fmaxf(t, s_tmp[w]);
  return t;
}

// One block per pair: the sums (Simpson sums scaled, |g|^2 raw, kept for the
// refinement), the FP32 score of every k < N with its error bound, and the
// candidates k whose score plus bound reaches the largest score minus bound.
constexpr int kCandBlock = 1024;  // few pairs leave the chip short of loads in flight otherwise
template <bool UN>
__global__ void __launch_bounds__(kCandBlock) k_mx_cand(const float2 *__restrict__ C, const double *__restrict__ part, int nblk, int N, int ld,
                          int ndet, const StreamDev *__restrict__ streams, const int *__restrict__ handles,
                          const int *__restrict__ req_status, double kscale, double *__restrict__ sums,
                          int *__restrict__ cand, int *__restrict__ ncand, int *__restrict__ overflow) {
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1;
  __shared__ float s_tmpf[kCandBlock / 32], s_scale[5];
  __shared__ int s_cnt;
  const int q = blockIdx.x, r = q / ndet;
  if (req_status && req_status[r]) {  // outside the model domain: no candidates, the result is NaN
    if (threadIdx.x == 0) ncand[q] = 0;
    return;
  }
  const StreamDev &st = streams[handles[q]];
  const double df = st.freqs[1] - st.freqs[0];
  // the sums and the scores' scales, on one warp (the FP64 pipe's time counts for
  // every warp that repeats them)
  if (threadIdx.x < 32) {
    double sm[NS];
#pragma unroll
    for (int j = 0; j < NS; j++) {
      double t = 0.0;
      for (int b = threadIdx.x; b < nblk; b += 32) t += part[((size_t)q * NS + j) * nblk + b];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      sm[j] = (UN ? j < 3 : j < 1) ? 4.0 * t * df / 3.0 : t;
    }
    if (threadIdx.x == 0) {
      for (int j = 0; j < NS; j++) sums[(size_t)q * NS + j] = sm[j];
      s_cnt = 0;
      if (UN) {
        const float I = (float)(sm[2] / (sqrt(sm[0]) * sqrt(sm[1])));
        const double ap = df / sqrt(sm[0]), ac = df / sqrt(sm[1]);
        s_scale[0] = (float)ap;
        s_scale[1] = (float)ac;
        s_scale[2] = I;
        s_scale[3] = (float)fmax((double)(float)ap * kTau * kscale * sqrt(sm[NS - 2]),
                                 (double)(float)ac * kTau * kscale * sqrt(sm[NS - 1]));
        s_scale[4] = 1.f / (1.f - fabsf(I));
      } else {
        s_scale[0] = (float)(kTau * kscale * sqrt(sm[1]));
      }
    }
  }
  // score and bound of bin k; the aligned form's bound is the same at every bin and
  // joins after the scan, which then does not wait for the sums
  if (UN) __syncthreads();
  const float ap = UN ? s_scale[0] : 0.f, ac = UN ? s_scale[1] : 0.f, I = UN ? s_scale[2] : 0.f,
              eps = UN ? s_scale[3] : 0.f, inv1mI = UN ? s_scale[4] : 0.f;
  float E = 0.f;
  auto score = [&](int k, float &lo, float &hi) {
    if (!UN) {
      const float2 v = C[(size_t)q * ld + k];
      const float m = sqrtf(v.x * v.x + v.y * v.y);
      lo = m - E;
      hi = m + E;
    } else {
      const float2 a = C[((size_t)q * NP) * ld + k], c = C[((size_t)q * NP + 1) * ld + k];
      const float rpx = ap * a.x, rpy = ap * a.y, rcx = ac * c.x, rcy = ac * c.y;
      const float p2 = rpx * rpx + rpy * rpy, c2 = rcx * rcx + rcy * rcy, gam = rpx * rcx + rpy * rcy;
      const float lam =
          (p2 + c2 - 2.f * gam * I + sqrtf(fmaxf((p2 - c2) * (p2 - c2) + 4.f * (I * p2 - gam) * (I * c2 - gam), 0.f))) /
          (1.f - I * I);
      // |d lambda| <= (4 (|rho+| + |rhox|) eps + 4 eps^2) / (1 - |I|), doubled, plus FP32 rounding of lambda
      const float D = 2.f * (4.f * (sqrtf(p2) + sqrtf(c2) + 2.f * eps) * eps + 4.f * eps * eps) * inv1mI +
                      1e-5f * fabsf(lam);
      lo = lam - D;
      hi = lam + D;
    }
  };
  float L = -INFINITY, H = -INFINITY;  // H: the largest upper bound of this thread's bins
  bool nan = false;
#pragma unroll 4
  for (int k = threadIdx.x; k < N; k += blockDim.x) {
    float lo, hi;
    score(k, lo, hi);
    L = fmaxf(L, lo);
    H = fmaxf(H, hi);
    nan = nan || hi != hi;
  }
  L = block_max(L, s_tmpf);
  if (!UN) {
    E = s_scale[0];
    L -= E;
    H += E;
  }
  if (H >= L || nan)
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
      float lo, hi;
      score(k, lo, hi);
      if (hi >= L || hi != hi) {  // NaN scores are candidates too
        const int i = atomicAdd(&s_cnt, 1);
        if (i < kCand) cand[(size_t)q * kCand + i] = k;
      }
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    ncand[q] = min(s_cnt, kCand);
    if (s_cnt > kCand) atomicExch(overflow, 1);
  }
}

// Fewer candidates for the refinement (two-float rows): the direct sum of each in
// FP32, four at a time so that a row is read once for them, groups of 16 products
// joining a two-float total.  Bounds of a part's error in units of 2^-24 ||g||_1:
// the 32 roundings of a group 32, its twiddles (within 2^-22 in each part) 4
// sqrt(2) = 5.7, the rows' and the total's low words 1.4 each, the last product's
// roundings 2 and twiddle 5.7: 48.2, and |G_k| is off by at most sqrt(2) times
// that.  So 72 2^-24 sqrt(N) ||g||_2 holds every |G_k|'s error -- a tenth of the
// transform's bound at most -- and the same interval test leaves those that may
// still be the maximum.  One block per pair; pairs with one candidate have nothing to do.
constexpr int kScreen = 4, kScreenBlock = 1024;
template <bool UN>
__global__ void __launch_bounds__(kScreenBlock, 1) k_mx_screen(const gwt::ff4 *__restrict__ rows,
                                                      const gwt::AccReq *__restrict__ areq, int ndet, int N,
                                                      const StreamDev *__restrict__ streams,
                                                      const int *__restrict__ handles, const double *__restrict__ sums,
                                                      const int *__restrict__ overflow, int *__restrict__ cand,
                                                      int *__restrict__ ncand) {
  using namespace gwt;
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1;
  extern __shared__ float2 s_tw[];  // [kScreen][nj]
  if (*overflow) return;  // the batch goes to the FP64 transforms
  __shared__ double s_part[kScreen * NP * 2][kScreenBlock / 32];
  __shared__ float s_lo[kCand], s_hi[kCand];
  __shared__ int s_k[kCand], s_keep;
  const int q = blockIdx.x, tid = threadIdx.x, bin = tid % kBlock, nc = ncand[q];
  if (nc <= 1) return;
  const StreamDev &st = streams[handles[q]];
  const int nl = live_bins(areq[q / ndet], streams[handles[q - q % ndet]].n0, N), nj = (N + kBlock - 1) / kBlock;
  if (tid < nc) s_k[tid] = cand[(size_t)q * kCand + tid];
  if (tid == 0) s_keep = 0;
  auto twiddle = [&](unsigned long long m) {  // e^{-2 pi i m / N}, m < N
    float s, c;
    q64_sincospi(((m << 32) / (unsigned)N) << 32, &s, &c);
    return make_float2(c, -s);
  };
  const double *sm = sums + (size_t)q * NS;
  const double unit = 72.0 / 16777216.0 * sqrt((double)N);
  for (int c0 = 0; c0 < nc; c0 += kScreen) {
    const int mc = min(kScreen, nc - c0);
    __syncthreads();
    for (int e = tid; e < mc * nj; e += kScreenBlock) {
      const int c = e / nj, j = e - c * nj;
      s_tw[e] = twiddle(((unsigned long long)j * kBlock % N) * s_k[c0 + c] % N);
    }
    __syncthreads();
    ff tot[kScreen * NP * 2];
#pragma unroll
    for (int u = 0; u < kScreen * NP * 2; u++) tot[u] = ff{0.f, 0.f};
    const ff4 *row = rows + (size_t)q * NP * N;
    for (int j0 = tid / kBlock * 16; j0 * kBlock < nl; j0 += kScreenBlock / kBlock * 16) {
      float a[kScreen * NP * 2];
#pragma unroll
      for (int u = 0; u < kScreen * NP * 2; u++) a[u] = 0.f;
#pragma unroll 8
      for (int j = j0; j < j0 + 16; j++) {
        const int n = j * kBlock + bin;
        const bool in = n < nl;
#pragma unroll
        for (int p = 0; p < NP; p++) {
          const ff4 x = in ? acc_ld(row + (size_t)p * N + n) : ff4{0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int c = 0; c < kScreen; c++) {
            const float2 w = s_tw[in && c < mc ? c * nj + j : 0];
            float &re = a[(c * NP + p) * 2], &im = a[(c * NP + p) * 2 + 1];
            re = fmaf(x.ch, w.x, fmaf(-x.sh, w.y, re));
            im = fmaf(x.ch, w.y, fmaf(x.sh, w.x, im));
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kScreen * NP * 2; u++) ff_acc(tot[u], ff{a[u], 0.f});
    }
#pragma unroll
    for (int c = 0; c < kScreen; c++) {
      const float2 w = twiddle(c < mc ? (unsigned long long)bin * s_k[c0 + c] % N : 0);
#pragma unroll
      for (int p = 0; p < NP; p++) {
        const ff re = tot[(c * NP + p) * 2], im = tot[(c * NP + p) * 2 + 1];
        ff v[2] = {two_sum(fmaf(re.h, w.x, -(im.h * w.y)), 0.f), two_sum(fmaf(re.h, w.y, im.h * w.x), 0.f)};
#pragma unroll
        for (int u = 0; u < 2; u++) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
            v[u] = ff_add(v[u], ff{__shfl_xor_sync(0xffffffffu, v[u].h, o), __shfl_xor_sync(0xffffffffu, v[u].l, o)});
          if ((tid & 31) == 0) s_part[(c * NP + p) * 2 + u][tid >> 5] = ff_value(v[u]);
        }
      }
    }
    __syncthreads();
    if (tid < mc) {
      double G[NP * 2];
#pragma unroll
      for (int u = 0; u < NP * 2; u++) {
        G[u] = 0.0;
        for (int w = 0; w < kScreenBlock / 32; w++) G[u] += s_part[tid * NP * 2 + u][w];
      }
      double lo, hi;
      if (!UN) {
        const double mag = sqrt(G[0] * G[0] + G[1] * G[1]), E = unit * sqrt(sm[1]);
        lo = mag - E;
        hi = mag + E;
      } else {
        const double df = st.freqs[1] - st.freqs[0], ap = df / sqrt(sm[0]), ac = df / sqrt(sm[1]);
        const double I = sm[2] / (sqrt(sm[0]) * sqrt(sm[1]));
        const double eps = fmax(ap * unit * sqrt(sm[3]), ac * unit * sqrt(sm[4]));
        const double rpx = ap * G[0], rpy = ap * G[1], rcx = ac * G[NP * 2 - 2], rcy = ac * G[NP * 2 - 1];
        const double p2 = rpx * rpx + rpy * rpy, c2 = rcx * rcx + rcy * rcy, gam = rpx * rcx + rpy * rcy;
        const double lam = (p2 + c2 - 2 * gam * I +
                            sqrt(fmax((p2 - c2) * (p2 - c2) + 4. * (I * p2 - gam) * (I * c2 - gam), 0.0))) / (1. - I * I);
        // k_mx_cand's bound on lambda with this error
        const double D = 2. * (4. * (sqrt(p2) + sqrt(c2) + 2. * eps) * eps + 4. * eps * eps) / (1. - fabs(I)) +
                         1e-5 * fabs(lam);
        lo = lam - D;
        hi = lam + D;
      }
      // outward to FP32
      s_lo[c0 + tid] = (float)lo - fabsf((float)lo) * 2.4e-7f;
      s_hi[c0 + tid] = (float)hi + fabsf((float)hi) * 2.4e-7f;
    }
  }
  __syncthreads();
  if (tid < nc) {
    float L = -INFINITY;
    for (int c = 0; c < nc; c++) L = fmaxf(L, s_lo[c]);
    if (!(s_hi[tid] < L)) cand[(size_t)q * kCand + atomicAdd(&s_keep, 1)] = s_k[tid];
  }
  __syncthreads();
  if (tid == 0) ncand[q] = s_keep;
}

// G_k of the candidate rows exactly in FP64: sum_n g_n e^{-2 pi i nk/N}, the
// twiddle of n = 256 j + i as e^{-2 pi i (256 j k mod N)/N} e^{-2 pi i (i k mod N)/N}
// (both phases reduced exactly in integers).  candval = |G_k|^2 (aligned) or
// lambda (unaligned).  Persistent over the (pair, candidate) slots.
template <bool UN>
__global__ void k_mx_refine(const double2 *__restrict__ g64, int N, int pairs, const int *__restrict__ cand,
                            const int *__restrict__ ncand, const int *__restrict__ overflow,
                            const double *__restrict__ sums, const StreamDev *__restrict__ streams,
                            const int *__restrict__ handles, double *__restrict__ candval) {
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1, NV = UN ? 4 : 2;
  extern __shared__ double2 s_wj[];
  if (*overflow) return;
  __shared__ double s_red[NV][kWarps];
  const int nj = (N + kBlock - 1) / kBlock;
  // slot s = (candidate ci, pair q) with ci major, so that the first
  // candidates of all pairs take consecutive blocks
  for (int sl = blockIdx.x; sl < pairs * kCand; sl += gridDim.x) {
    const int q = sl % pairs, ci = sl / pairs, it = q * kCand + ci;
    if (ci >= ncand[q]) continue;
    const long long k = cand[it];
    __syncthreads();  // the previous slot's table has been read
    for (int j = threadIdx.x; j < nj; j += blockDim.x) {
      const long long t = ((long long)j * kBlock % N) * k % N;
      double sn, cs;
      sincospi(2.0 * (double)t / (double)N, &sn, &cs);
      s_wj[j] = make_double2(cs, -sn);
    }
    double2 wi;
    {
      const long long t = (long long)threadIdx.x * k % N;
      double sn, cs;
      sincospi(2.0 * (double)t / (double)N, &sn, &cs);
      wi = make_double2(cs, -sn);
    }
    __syncthreads();
    double v[NV];
#pragma unroll
    for (int u = 0; u < NV; u++) v[u] = 0.0;
    // this thread's bins n = 256 j + i: sum_j g_n e^{-2 pi i 256 j k/N}, then
    // one product with e^{-2 pi i i k/N}
    const double2 *row = g64 + ((size_t)q * NP) * N;
    for (int j = 0; j < nj; j++) {
      const int n = j * kBlock + threadIdx.x;
      if (n >= N) break;
      const double2 w = s_wj[j];
      const double2 x = row[n];
      v[0] += x.x * w.x - x.y * w.y;
      v[1] += x.x * w.y + x.y * w.x;
      if (UN) {
        const double2 y = row[N + n];
        v[2] += y.x * w.x - y.y * w.y;
        v[3] += y.x * w.y + y.y * w.x;
      }
    }
#pragma unroll
    for (int u = 0; u < NV; u += 2) {
      const double re = v[u] * wi.x - v[u + 1] * wi.y, im = v[u] * wi.y + v[u + 1] * wi.x;
      v[u] = re;
      v[u + 1] = im;
    }
#pragma unroll
    for (int u = 0; u < NV; u++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[u] += __shfl_xor_sync(0xffffffffu, v[u], o);
    }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int u = 0; u < NV; u++) s_red[u][threadIdx.x >> 5] = v[u];
    __syncthreads();
    if (threadIdx.x == 0) {
      double G[NV];
#pragma unroll
      for (int u = 0; u < NV; u++) {
        G[u] = 0.0;
        for (int w = 0; w < kWarps; w++) G[u] += s_red[u][w];
      }
      if (!UN) {
        candval[it] = G[0] * G[0] + G[1] * G[1];
      } else {
        const double *sm = sums + (size_t)q * NS;
        const StreamDev &st = streams[handles[q]];
        const double df = st.freqs[1] - st.freqs[0];
        const double ap = df / sqrt(sm[0]), ac = df / sqrt(sm[1]);
        const double I = sm[2] / (sqrt(sm[0]) * sqrt(sm[1]));
        const double rpx = ap * G[0], rpy = ap * G[1], rcx = ac * G[2], rcy = ac * G[3];
        const double p2 = rpx * rpx + rpy * rpy, c2 = rcx * rcx + rcy * rcy, gam = rpx * rcx + rpy * rcy;
        candval[it] =
            (p2 + c2 - 2 * gam * I + sqrt((p2 - c2) * (p2 - c2) + 4. * (I * p2 - gam) * (I * c2 - gam))) / (1. - I * I);
      }
    }
  }
}

// k_mx_refine on two-float rows: the twiddles from their exact fixed-point turns,
// products and sums in two floats, bins beyond the cut left out.  A candidate or two
// per pair have work, a few per SM: a block takes two rows of 256 bins at a time, so
// that the last ones end together, and a thread keeps eight loads in flight (384
// rows of 32,128 bins: 46 us; blocks of 256 threads, two an SM, 71).
constexpr int kRefineBlock = 512;
template <bool UN>
__global__ void __launch_bounds__(kRefineBlock, 2) k_mx_refine_ff(const gwt::ff4 *__restrict__ rows,
                                                         const gwt::AccReq *__restrict__ areq, int ndet,
                                                         const gwt::AccLut *__restrict__ glut, int N, int pairs,
                                                         const int *__restrict__ cand, const int *__restrict__ ncand,
                                                         const int *__restrict__ overflow,
                                                         const double *__restrict__ sums,
                                                         const StreamDev *__restrict__ streams,
                                                         const int *__restrict__ handles, double *__restrict__ candval) {
  using namespace gwt;
  constexpr int NS = UN ? 5 : 2, NP = UN ? 2 : 1, NV = 2 * NP;
  extern __shared__ double2 s_wj[];
  ff4 *s_wf = (ff4 *)s_wj, *s_turn = s_wf + (N + kBlock - 1) / kBlock;
  __shared__ double s_red[NV][kRefineBlock / 32];
  constexpr int kLoads = UN ? 4 : 8;  // in flight per thread
  if (*overflow) return;
  const int nj = (N + kBlock - 1) / kBlock, tid = threadIdx.x, bin = tid % kBlock;
  bool loaded = false;
  for (int sl = blockIdx.x; sl < pairs * kCand; sl += gridDim.x) {
    const int q = sl % pairs, ci = sl / pairs, it = q * kCand + ci;
    if (ci >= ncand[q]) continue;
    const unsigned k = (unsigned)cand[it];
    __syncthreads();  // the previous slot's table has been read
    if (!loaded) {
      for (int w = tid; w < kTurnTab; w += kRefineBlock) s_turn[w] = acc_ld(glut->turn + w);
      __syncthreads();
      loaded = true;
    }
    auto twiddle = [&](unsigned long long m, ff &c, ff &s) {  // e^{-2 pi i m / N}, m < N: m / N 2^64 in two quotients
      const unsigned long long a = (m << 32) / (unsigned)N, rem = (m << 32) - a * (unsigned)N;
      ff_turns_sincos(0ull - ((a << 32) + (rem << 32) / (unsigned)N), s_turn, c, s);
    };
    for (int j = tid; j < nj; j += kRefineBlock) {
      ff c, s;
      twiddle(((unsigned long long)j * kBlock % N) * k % N, c, s);
      s_wf[j] = ff4{c.h, c.l, s.h, s.l};
    }
    ff wc, ws;
    twiddle((unsigned long long)bin * k % N, wc, ws);
    __syncthreads();
    const int nl = live_bins(areq[q / ndet], streams[handles[q - q % ndet]].n0, N);
    const ff4 *row = rows + ((size_t)q * NP) * N;
    // this thread's bins n = 256 j + i: sum_j g_n e^{-2 pi i 256 j k/N}, then
    // one product with e^{-2 pi i i k/N}
    ff v[NV];
#pragma unroll
    for (int u = 0; u < NV; u++) v[u] = ff{0.f, 0.f};
    for (int j0 = tid / kBlock * kLoads; j0 * kBlock < nl; j0 += kRefineBlock / kBlock * kLoads) {
      ff4 x[kLoads][NP];
#pragma unroll
      for (int j = 0; j < kLoads; j++) {
        const int n = (j0 + j) * kBlock + bin;
#pragma unroll
        for (int u = 0; u < NP; u++) x[j][u] = n < nl ? acc_ld(row + (size_t)u * N + n) : ff4{0.f, 0.f, 0.f, 0.f};
      }
#pragma unroll
      for (int j = 0; j < kLoads; j++) {
        const ff4 w = s_wf[j0 + j < nj ? j0 + j : 0];
        const ff wr{w.ch, w.cl}, wi{w.sh, w.sl};
#pragma unroll
        for (int u = 0; u < NP; u++) {
          const ff xr{x[j][u].ch, x[j][u].cl}, xi{x[j][u].sh, x[j][u].sl};
          ff_acc(v[2 * u], ff_sub(ff_mul(xr, wr), ff_mul(xi, wi)));
          ff_acc(v[2 * u + 1], ff_add(ff_mul(xr, wi), ff_mul(xi, wr)));
        }
      }
#pragma unroll
      for (int u = 0; u < NV; u++) v[u] = ff_norm(v[u]);  // the low part stays an ulp of the sum
    }
#pragma unroll
    for (int u = 0; u < NV; u += 2) {
      ff p[2] = {ff_norm(ff_sub(ff_mul(v[u], wc), ff_mul(v[u + 1], ws))),
                 ff_norm(ff_add(ff_mul(v[u], ws), ff_mul(v[u + 1], wc)))};
#pragma unroll
      for (int e = 0; e < 2; e++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          p[e] = ff_add(p[e], ff{__shfl_xor_sync(0xffffffffu, p[e].h, o), __shfl_xor_sync(0xffffffffu, p[e].l, o)});
        if ((tid & 31) == 0) s_red[u + e][tid >> 5] = ff_value(p[e]);
      }
    }
    __syncthreads();
    if (tid == 0) {
      double G[NV];
#pragma unroll
      for (int u = 0; u < NV; u++) {
        G[u] = 0.0;
        for (int w = 0; w < kRefineBlock / 32; w++) G[u] += s_red[u][w];
      }
      if (!UN) {
        candval[it] = G[0] * G[0] + G[1] * G[1];
      } else {
        const double *sm = sums + (size_t)q * NS;
        const StreamDev &st = streams[handles[q]];
        const double df = st.freqs[1] - st.freqs[0];
        const double ap = df / sqrt(sm[0]), ac = df / sqrt(sm[1]);
        const double I = sm[2] / (sqrt(sm[0]) * sqrt(sm[1]));
        const double rpx = ap * G[0], rpy = ap * G[1], rcx = ac * G[NV - 2], rcy = ac * G[NV - 1];
        const double p2 = rpx * rpx + rpy * rpy, c2 = rcx * rcx + rcy * rcy, gam = rpx * rcx + rpy * rcy;
        candval[it] =
            (p2 + c2 - 2 * gam * I + sqrt((p2 - c2) * (p2 - c2) + 4. * (I * p2 - gam) * (I * c2 - gam))) / (1. - I * I);
      }
    }
  }
}

// One thread per request: log L of each pair from its best candidate, summed
// over the detectors in order.
template <bool UN>
__global__ void k_mx_final(const double *__restrict__ candval, const int *__restrict__ ncand,
                           const double *__restrict__ sums, int n, int ndet, const StreamDev *__restrict__ streams,
                           const int *__restrict__ handles, const int *__restrict__ req_status,
                           double *__restrict__ out, int *__restrict__ status) {
  constexpr int NS = UN ? 5 : 2;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int rs = req_status ? req_status[r] : 0;
  double ll = 0.0;
  for (int d = 0; d < ndet; d++) {
    const int q = r * ndet + d;
    double mx = -HUGE_VAL;
    for (int c = 0; c < ncand[q]; c++) mx = fmax(mx, candval[(size_t)q * kCand + c]);
    if (UN) {
      ll += 0.25 * mx;
    } else {
      const StreamDev &st = streams[handles[q]];
      const double df = st.freqs[1] - st.freqs[0];
      ll += 0.5 * (mx * df * df) / sums[(size_t)q * NS];
    }
  }
  out[r] = rs ? __longlong_as_double(0x7ff8000000000000ll) : ll;
  if (status) status[r] = rs;
}

// max |B_j| over the Bluestein kernel (one block).
__global__ void k_absmax(const double2 *__restrict__ B, int M, double *__restrict__ out) {
  __shared__ double s[kWarps];
  double m = 0.0;
  for (int i = threadIdx.x; i < M; i += blockDim.x) m = fmax(m, hypot(B[i].x, B[i].y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = s[0];
    for (int w = 1; w < kWarps; w++) t = fmax(t, s[w]);
    *out = t;
  }
}

__global__ void k_to_f32(const double2 *__restrict__ x, float2 *__restrict__ y, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = make_float2((float)x[i].x, (float)x[i].y);
}

size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

bool smooth7(int n) {
  for (int p : {2, 3, 5, 7})
    while (n % p == 0) n /= p;
  return n == 1;
}

// Transform length: N itself when cuFFT handles it directly, else the
// Bluestein power of two M >= 2N - 1.
int xform_len(int N, int *blue) {
  *blue = !smooth7(N);
  if (!*blue) return N;
  int M = 1;
  while (M < 2 * N - 1) M <<= 1;
  return M;
}

// The Bluestein kernel for N, FFT_M(b)/M in FP64 (kWsChirp) and FP32
// (kWsChirp32), and the search's error scale M max|B|, kept until N changes; in
// FP32 also the chirp, and conv.cu's tables (*conv; null where it has no kernels
// for M or there is no memory for them).
int ensure_chirp(gwgpu_context *c, int N, int M, const double2 **B64, const float2 **B32, const float2 **tab,
                 void **conv = nullptr) {
  void *kb, *kb32;
  const size_t b32 = up256(8 * ((size_t)M + N)), bconv = gwk::conv_table_bytes(M);
  // a workspace that grows loses what it held, also when a later step fails
  const bool have = c->chirp_n == N;
  if (!have) c->chirp_n = 0;
  int st = c->workspace(gwgpu_context::kWsChirp, 16 * (size_t)M + 256, &kb);
  if (st) return st;
  if (!have) c->chirp_conv = bconv && c->workspace(gwgpu_context::kWsChirp32, b32 + bconv, &kb32) == GWGPU_OK;
  if ((st = c->workspace(gwgpu_context::kWsChirp32, b32 + (c->chirp_conv ? bconv : 0), &kb32))) return st;
  *B64 = (const double2 *)kb;
  *B32 = (const float2 *)kb32;
  *tab = *B32 + M;
  if (conv) *conv = c->chirp_conv ? (char *)kb32 + b32 : nullptr;
  if (have) return GWGPU_OK;
  int p1;
  if ((st = gwfft::plan(c, gwfft::kZ2Z, M, 1, &p1))) return st;
  const int gb = std::min((M + kBlock - 1) / kBlock, 1024);
  k_chirp_fill<<<gb, kBlock, 0, c->stream>>>((double2 *)kb, N, M);
  if ((st = gwfft::exec_z2z(c, p1, (double2 *)kb, (double2 *)kb, gwfft::kForward, c->stream))) return st;
  double *dmax = (double *)((char *)kb + 16 * (size_t)M);
  k_absmax<<<1, kBlock, 0, c->stream>>>((const double2 *)kb, M, dmax);
  k_to_f32<<<gb, kBlock, 0, c->stream>>>((const double2 *)kb, (float2 *)kb32, M);
  k_chirp_tab<<<gb, kBlock, 0, c->stream>>>((float2 *)kb32 + M, N);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && c->chirp_conv)
    e = gwk::launch_conv_tables((const float2 *)kb32, M, (char *)kb32 + b32, c->stream);
  if (e != cudaSuccess) return c->fail(e, "Bluestein kernel");
  double bmax = 0;
  cudaMemcpyAsync(&bmax, dmax, 8, cudaMemcpyDeviceToHost, c->stream);
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->fail(e, "Bluestein kernel");
  c->chirp_kscale = (double)M * bmax;
  c->chirp_n = N;
  return GWGPU_OK;
}

// What both entry points hand to the pipeline (device pointers).
struct MxIn {
  const Request *req = nullptr;               // requests (intrinsic mode), or null
  const gwt::AccReq *areq = nullptr;          // the same for the search on two-float bins, or null
  const double2 *rp = nullptr, *rc = nullptr;  // responses per pair, rows of N, when req is null
  const StreamDev *streams = nullptr;
  const int *handles = nullptr;                // [n * ndet]
  const int *req_status = nullptr;             // per request, or null
  int n = 0, ndet = 0, N = 0;
  bool un = false;
  bool search = true;                          // false: a search has given up on these requests
  // the results and the search's overflow flag (*overflow, on the host at
  // *h_overflow once copied) go to the host in one copy
  void *results = nullptr, *h_results = nullptr;
  size_t result_bytes = 0;
  int *overflow = nullptr;
  const volatile int *h_overflow = nullptr;
};

// The FP64 transforms: prep, FFT_M (Bluestein) or FFT_N, reduction.
int run_fp64(gwgpu_context *c, const MxIn &in, double *out, int *status) {
  const int np = in.un ? 2 : 1, ns = in.un ? 3 : 1, pairs = in.n * in.ndet, rows = pairs * np;
  int blue;
  const int ld = xform_len(in.N, &blue);
  const double2 *B64 = nullptr;
  const float2 *B32 = nullptr;
  const float2 *ctab = nullptr;
  int st = blue ? ensure_chirp(c, in.N, ld, &B64, &B32, &ctab) : GWGPU_OK;
  if (st) return st;
  int plan;  // fetched last: a new plan may reset the cache (cufft_rt.cu)
  if ((st = gwfft::plan(c, gwfft::kZ2Z, ld, rows, &plan))) return st;
  const int nblk = (ld + kBlock - 1) / kBlock;
  const size_t o_g = 0, o_h = up256(16 * (size_t)rows * ld), o_ll = o_h + up256(8 * (size_t)pairs * ns * nblk),
               o_done = o_ll + up256(8 * (size_t)pairs), total = o_done + up256(4 * (size_t)in.n);
  void *dev;
  if ((st = c->workspace(gwgpu_context::kWsMaxllRun, total, &dev))) return st;
  char *b = (char *)dev;
  double2 *g = (double2 *)(b + o_g);
  double *hh = (double *)(b + o_h);
  unsigned *done = (unsigned *)(b + o_done);
  cudaMemsetAsync(done, 0, 4 * (size_t)in.n, c->stream);
  const dim3 grid(nblk, in.n);
  if (in.un)
    k_maxll_prep<true><<<grid, kBlock, 0, c->stream>>>(in.req, in.rp, in.rc, in.ndet, in.streams, in.handles, in.N,
                                                        ld, blue, g, hh);
  else
    k_maxll_prep<false><<<grid, kBlock, 0, c->stream>>>(in.req, in.rp, in.rc, in.ndet, in.streams, in.handles, in.N,
                                                         ld, blue, g, hh);
  if ((st = gwfft::exec_z2z(c, plan, g, g, gwfft::kForward, c->stream))) return st;
  if (blue) {
    const long long tot = (long long)rows * ld;
    const int gb = (int)std::min<long long>((tot + kBlock - 1) / kBlock, 152 * 16);
    k_chirp_mul<<<gb, kBlock, 0, c->stream>>>(g, B64, ld, tot);
    if ((st = gwfft::exec_z2z(c, plan, g, g, gwfft::kInverse, c->stream))) return st;
  }
  if (in.un)
    k_maxll_reduce<true><<<pairs, kBlock, 0, c->stream>>>(g, hh, nblk, in.N, ld, in.ndet, in.streams, in.handles,
                                                          in.req_status, (double *)(b + o_ll), done, out, status);
  else
    k_maxll_reduce<false><<<pairs, kBlock, 0, c->stream>>>(g, hh, nblk, in.N, ld, in.ndet, in.streams, in.handles,
                                                           in.req_status, (double *)(b + o_ll), done, out, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GWGPU_OK : c->fail(e, "maximised likelihood launch");
}

// The FP32 search and its refinement; *fallback set when a pair had more
// candidates than kCand, or the two-float arrays gave way to an allocation
// (nothing written to out then).  128 IMRPhenomD requests
// on 3 x 32,128 bins, device time by kernel: products 97, transforms and chirp
// 209 (conv.cu; 434 with library transforms), candidates 55 (132 with its FP64 sums on every warp), screen 31 and
// two-float refinement 46 (389 for FP64 sums of every candidate over the whole
// row), result 9 us; one copy each way through pinned memory and one
// synchronisation at the end: the overflow flag travels with the results.
int run_search(gwgpu_context *c, const MxIn &in, double *out, int *status, bool *fallback) {
  const int np = in.un ? 2 : 1, ns = in.un ? 5 : 2, pairs = in.n * in.ndet, rows = pairs * np;
  *fallback = false;
  int blue;
  const int ld = xform_len(in.N, &blue);
  const double2 *B64 = nullptr;
  const float2 *B32 = nullptr, *ctab = nullptr;
  double kscale = std::sqrt((double)in.N);
  int st = GWGPU_OK;
  void *conv = nullptr;
  if (blue) {
    if ((st = ensure_chirp(c, in.N, ld, &B64, &B32, &ctab, &conv))) return st;
    kscale = c->chirp_kscale;
  }
  int plan = 0;  // fetched last: a new plan may reset the cache (cufft_rt.cu)
  if (!conv && (st = gwfft::plan(c, gwfft::kC2C, ld, rows, &plan))) return st;
  const bool two = in.areq != nullptr;  // two-float bins
  const int pad = conv ? in.N : ld, per = two ? kPrepTile : kBlock, nblk = (pad + per - 1) / per;
  const size_t o_g = 0, o_a = up256(16 * (size_t)rows * in.N), o_h = o_a + up256(8 * (size_t)rows * ld),
               o_s = o_h + up256(8 * (size_t)pairs * ns * nblk), o_c = o_s + up256(8 * (size_t)pairs * ns),
               o_nc = o_c + up256(4 * (size_t)pairs * kCand), o_v = o_nc + up256(4 * (size_t)pairs),
               total = o_v + up256(8 * (size_t)pairs * kCand);
  void *dev;
  if ((st = c->workspace(gwgpu_context::kWsMaxllRun, total, &dev))) return st;
  if (two && c->two_float_off) {
    *fallback = true;
    return GWGPU_OK;
  }
  char *b = (char *)dev;
  double2 *g64 = (double2 *)(b + o_g);
  float2 *a32 = (float2 *)(b + o_a);
  double *hh = (double *)(b + o_h), *sums = (double *)(b + o_s), *cv = (double *)(b + o_v);
  int *cand = (int *)(b + o_c), *ncand = (int *)(b + o_nc), *ovf = in.overflow;
  cudaMemsetAsync(ovf, 0, 4, c->stream);
  const dim3 grid(nblk, in.n);
  if (two && in.un)
    k_mx_prep_ff<true><<<grid, kBlock, 0, c->stream>>>(in.areq, in.ndet, in.streams, in.handles, c->acc, c->acc_lut,
                                                        in.N, ld, pad, blue, ctab, (gwt::ff4 *)g64, a32, hh);
  else if (two)
    k_mx_prep_ff<false><<<grid, kBlock, 0, c->stream>>>(in.areq, in.ndet, in.streams, in.handles, c->acc, c->acc_lut,
                                                         in.N, ld, pad, blue, ctab, (gwt::ff4 *)g64, a32, hh);
  else if (in.un)
    k_mx_prep<true><<<grid, kBlock, 0, c->stream>>>(in.req, in.rp, in.rc, in.ndet, in.streams, in.handles, in.N, ld,
                                                     blue, g64, a32, hh);
  else
    k_mx_prep<false><<<grid, kBlock, 0, c->stream>>>(in.req, in.rp, in.rc, in.ndet, in.streams, in.handles, in.N, ld,
                                                      blue, g64, a32, hh);
  if (conv) {
    cudaError_t ce = gwk::launch_conv(a32, rows, in.N, ld, gwk::conv_tables_at(conv, ld), c->stream);
    if (ce != cudaSuccess) return c->fail(ce, "maximised likelihood transform");
  } else if ((st = gwfft::exec_c2c(c, plan, a32, a32, gwfft::kForward, c->stream))) {
    return st;
  }
  if (blue && !conv) {
    const long long tot = (long long)rows * ld;
    const int gb = (int)std::min<long long>((tot + kBlock - 1) / kBlock, 152 * 16);
    k_chirp_mul32<<<gb, kBlock, 0, c->stream>>>(a32, B32, ld, tot);
    if ((st = gwfft::exec_c2c(c, plan, a32, a32, gwfft::kInverse, c->stream))) return st;
  }
  if (in.un)
    k_mx_cand<true><<<pairs, kCandBlock, 0, c->stream>>>(a32, hh, nblk, in.N, ld, in.ndet, in.streams, in.handles,
                                                      in.req_status, kscale, sums, cand, ncand, ovf);
  else
    k_mx_cand<false><<<pairs, kCandBlock, 0, c->stream>>>(a32, hh, nblk, in.N, ld, in.ndet, in.streams, in.handles,
                                                       in.req_status, kscale, sums, cand, ncand, ovf);
  const int nj = (in.N + kBlock - 1) / kBlock;
  const size_t smem = 16 * (size_t)nj;
  const int gr = std::min(pairs * kCand, 152 * 8);
  if (two) {
    const size_t tw = sizeof(float2) * (size_t)kScreen * nj;
    auto screen = [&](auto kern) {
      if (tw > 48 * 1024) cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tw);
      kern<<<pairs, kScreenBlock, tw, c->stream>>>((const gwt::ff4 *)g64, in.areq, in.ndet, in.N, in.streams, in.handles,
                                              sums, ovf, cand, ncand);
    };
    if (tw <= 200 * 1024) {  // longer rows keep every candidate
      if (in.un) screen(k_mx_screen<true>);
      else screen(k_mx_screen<false>);
    }
  }
  auto refine = [&](auto kern) {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<gr, kBlock, smem, c->stream>>>(g64, in.N, pairs, cand, ncand, ovf, sums, in.streams, in.handles, cv);
  };
  const size_t smem_ff = smem + sizeof(gwt::ff4) * gwt::kTurnTab;
  auto refine_ff = [&](auto kern) {
    if (smem_ff > 48 * 1024)
      cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_ff);
    kern<<<gr, kRefineBlock, smem_ff, c->stream>>>((const gwt::ff4 *)g64, in.areq, in.ndet, c->acc_lut, in.N, pairs, cand,
                                             ncand, ovf, sums, in.streams, in.handles, cv);
  };
  if (two && in.un) refine_ff(k_mx_refine_ff<true>);
  else if (two) refine_ff(k_mx_refine_ff<false>);
  else if (in.un) refine(k_mx_refine<true>);
  else refine(k_mx_refine<false>);
  if (in.un)
    k_mx_final<true><<<(in.n + 127) / 128, 128, 0, c->stream>>>(cv, ncand, sums, in.n, in.ndet, in.streams,
                                                                 in.handles, in.req_status, out, status);
  else
    k_mx_final<false><<<(in.n + 127) / 128, 128, 0, c->stream>>>(cv, ncand, sums, in.n, in.ndet, in.streams,
                                                                  in.handles, in.req_status, out, status);
  // with a pair of too many candidates the screen and the refinement do nothing,
  // and the results are not used
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->fail(e, "maximised likelihood launch");
  cudaMemcpyAsync(in.h_results, in.results, in.result_bytes, cudaMemcpyDeviceToHost, c->stream);
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->fail(e, "maximised likelihood");
  *fallback = *in.h_overflow != 0;
  return GWGPU_OK;
}

bool search_fits(const gwgpu_context *c, int N) { return !c->maxll_fp64 && (N + kBlock - 1) / kBlock <= kMaxTwiddleRows; }

// The results on the host (in.h_results); *searched: false when only the FP64
// transforms' inputs (in.req) will do.
int maxll_run(gwgpu_context *c, const MxIn &in, double *out, int *status, bool *searched = nullptr) {
  if (searched) *searched = true;
  if (in.search && search_fits(c, in.N)) {
    bool fb = false;
    int st = run_search(c, in, out, status, &fb);
    if (st || !fb) return st;
  }
  if (in.areq && !in.req) {
    *searched = false;
    return GWGPU_OK;
  }
  int st = run_fp64(c, in, out, status);
  if (st) return st;
  cudaMemcpyAsync(in.h_results, in.results, in.result_bytes, cudaMemcpyDeviceToHost, c->stream);
  cudaError_t e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? GWGPU_OK : c->fail(e, "maximised likelihood");
}

// One pair from host arrays: hp (and hc when unaligned) given.
int maximized_single(gwgpu_context *c, const double *data, const double *psd, const double *freqs, const double *hp,
                     const double *hc, int N, double *out) {
  const bool un = hc != nullptr;
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const size_t o_f = 0, o_d = up256(8 * (size_t)N), o_s = o_d + up256(16 * (size_t)N),
               o_rp = o_s + up256(8 * (size_t)N), o_rc = o_rp + up256(16 * (size_t)N),
               o_sd = o_rc + up256(16 * (size_t)N), o_misc = o_sd + up256(sizeof(StreamDev)), total = o_misc + 256;
  void *dev;
  int st = c->workspace(gwgpu_context::kWsMaxll, total, &dev);
  if (st) return st;
  char *b = (char *)dev;
  cudaMemcpyAsync(b + o_f, freqs, 8 * (size_t)N, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(b + o_d, data, 16 * (size_t)N, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(b + o_s, psd, 8 * (size_t)N, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(b + o_rp, hp, 16 * (size_t)N, cudaMemcpyHostToDevice, c->stream);
  if (un) cudaMemcpyAsync(b + o_rc, hc, 16 * (size_t)N, cudaMemcpyHostToDevice, c->stream);
  StreamDev sd;
  std::memset(&sd, 0, sizeof(sd));
  sd.N = N;
  sd.freqs = (const double *)(b + o_f);
  sd.data = (const double *)(b + o_d);
  sd.psd = (const double *)(b + o_s);
  cudaMemcpyAsync(b + o_sd, &sd, sizeof(sd), cudaMemcpyHostToDevice, c->stream);
  int *dh = (int *)(b + o_misc);
  double *res = (double *)(b + o_misc + 64);
  cudaMemsetAsync(dh, 0, sizeof(int), c->stream);
  MxIn in;
  in.rp = (const double2 *)(b + o_rp);
  in.rc = un ? (const double2 *)(b + o_rc) : nullptr;
  in.streams = (const StreamDev *)(b + o_sd);
  in.handles = dh;
  in.n = 1;
  in.ndet = 1;
  in.N = N;
  in.un = un;
  double h[2];  // the result, the flag
  in.results = res;
  in.h_results = h;
  in.result_bytes = sizeof(h);
  in.overflow = (int *)(res + 1);
  in.h_overflow = (const int *)(h + 1);
  if ((st = maxll_run(c, in, res, nullptr))) return st;
  *out = h[0];
  return GWGPU_OK;
}

}  // namespace

extern "C" {

int gwgpu_maximized_log_likelihood_internal(gwgpu_context *c, const double *data, const double *psd,
                                            const double *freqs, const double *response, int N, double *out) {
  if (!c || !data || !psd || !freqs || !response || !out || N < 2) return GWGPU_EINVAL;
  return maximized_single(c, data, psd, freqs, response, nullptr, N, out);
}

int gwgpu_maximized_log_likelihood_unaligned_internal(gwgpu_context *c, const double *data, const double *psd,
                                                      const double *freqs, const double *hplus, const double *hcross,
                                                      int N, double *out) {
  if (!c || !data || !psd || !freqs || !hplus || !hcross || !out || N < 2) return GWGPU_EINVAL;
  return maximized_single(c, data, psd, freqs, hplus, hcross, N, out);
}

int gwgpu_maximized_loglik_batch(gwgpu_context *c, const gwgpu_gen_params *params, int n, int approximant,
                                 const int *handles, int ndet, double *loglik, int *status) {
  if (!c || !params || n < 1 || !handles || ndet < 1 || ndet > gwt::kMaxDet || !loglik) return GWGPU_EINVAL;
  if (approximant != GWGPU_IMRPHENOMD && approximant != GWGPU_IMRPHENOMPV2) return GWGPU_EINVAL;
  const bool un = approximant == GWGPU_IMRPHENOMPV2;
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const gwgpu_context::Stream *s0 = c->get_stream(handles[0]);
  if (!s0) return GWGPU_ENOTFOUND;
  const int N = s0->dev.N;
  for (int i = 0; i < n * ndet; i++) {
    const gwgpu_context::Stream *s = c->get_stream(handles[i]);
    if (!s) return GWGPU_ENOTFOUND;
    if (s->dev.N != N || s->dev.iw) {
      c->last_error = "maximised likelihood: one Simpson grid length for the whole batch";
      return GWGPU_EINVAL;
    }
  }
  const int pairs = n * ndet;
  const size_t o_p = 0, o_a = up256(sizeof(gwgpu_gen_params) * n), o_h = o_a + up256(4 * (size_t)n),
               o_req = o_h + up256(4 * (size_t)pairs),
               o_out = o_req + up256(std::max(sizeof(Request), sizeof(gwt::AccReq)) * n),
               o_st = o_out + 8 * (size_t)n, o_ovf = o_st + 4 * (size_t)n, total = o_ovf + 4;
  void *dev;
  int st = c->workspace(gwgpu_context::kWsMaxll, total, &dev);
  if (st) return st;
  char *b = (char *)dev;
  // inputs and results by one copy each through pinned memory
  char *h;
  if ((st = c->pinned(gwgpu_context::kHwsMaxll, o_req + total - o_out, (void **)&h))) return st;
  // the sampler's intrinsic mode fixes the extrinsic parameters
  // (IMRPhenomD: mcmc_gw.cpp:2614-2620, 2645-2651; IMRPhenomPv2: 2693-2699)
  gwgpu_gen_params *hp = (gwgpu_gen_params *)(h + o_p);
  for (int i = 0; i < n; i++) {
    gwgpu_gen_params &p = hp[i];
    p = params[i];
    p.RA = p.DEC = p.psi = 0;
    p.phiRef = 1;
    p.f_ref = un ? 20 : 10;
    p.incl_angle = 0;
    p.tc = 1;
    ((int *)(h + o_a))[i] = un ? gwt::kPhenomPv2 : gwt::kPhenomD;
  }
  std::memcpy(h + o_h, handles, 4 * (size_t)pairs);
  struct Drain {  // the pinned inputs are read by then, on every way out
    cudaStream_t s;
    ~Drain() {
      if (s) cudaStreamSynchronize(s);
    }
  } drain{c->stream};
  cudaMemcpyAsync(b, h, o_req, cudaMemcpyHostToDevice, c->stream);
  // two-float bins when every stream has its pairs; a search that gives up on
  // them leaves the FP64 transforms, which take the requests themselves
  bool two = c->acc_lut && search_fits(c, N) && N <= kBlock * (kMaxTwiddleRows - gwt::kTurnTab);
  for (int i = 0; i < pairs && two; i++) {
    const StreamDev &sd = c->get_stream(handles[i])->dev;
    two = sd.wd && sd.n0 + sd.N - 1 <= c->acc.nmax;
  }
  int *dst = (int *)(b + o_st);
  cudaError_t e;
  for (bool search = true;;) {
    e = gwk::launch_prologue((const gwt::GenParams *)(b + o_p), (const int *)(b + o_a), n, (const int *)(b + o_h),
                             ndet, 0.0, 0, c->streams_dev, c->qnm_dev, two ? nullptr : (Request *)(b + o_req), nullptr,
                             0, dst, c->stream, gwk::OrderArgs(), two ? (gwt::AccReq *)(b + o_req) : nullptr);
    if (e != cudaSuccess) return c->fail(e, "maximised likelihood prologue");
    MxIn in;
    if (two) in.areq = (const gwt::AccReq *)(b + o_req);
    else in.req = (const Request *)(b + o_req);
    in.streams = c->streams_dev;
    in.handles = (const int *)(b + o_h);
    in.req_status = dst;
    in.n = n;
    in.ndet = ndet;
    in.N = N;
    in.un = un;
    in.search = search;
    in.results = b + o_out;
    in.h_results = h + o_req;
    in.result_bytes = total - o_out;
    in.overflow = (int *)(b + o_ovf);
    in.h_overflow = (const int *)(h + o_req + (o_ovf - o_out));
    bool searched = true;
    if ((st = maxll_run(c, in, (double *)(b + o_out), dst, &searched))) return st;
    if (searched) break;
    search = search && c->two_float_off;  // no search yet where the two-float arrays gave way
    two = false;
  }
  drain.s = nullptr;
  std::memcpy(loglik, h + o_req, 8 * (size_t)n);
  const int *hs = (const int *)(h + o_req + (o_st - o_out));
  if (status)
    for (int i = 0; i < n; i++) status[i] = gwk::status_code(hs[i]);
  return GWGPU_OK;
}

}  // extern "C"

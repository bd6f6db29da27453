// fisher.cu -- numerical Fisher matrices (fisher.cpp:81-557, 2704-2781).
//
// Plain form (gwgpu_fisher_numerical): the reference algorithm for one source
// and one detector -- complex central differences of the FP64 detector
// response at theta +- eps (one-sided at eta = 1/4), DTOA phase factor for a
// non-reference detector, log-factor chain rule, then the Simpson Gram matrix.
//
// Batched form (gwgpu_fisher_batch): many sources x detectors in one pass.
// The same central differences are taken of the FP64 amplitude A and phase
// Phi separately and combined at the centre,
//   d r_d = e^{-i Psi_d} (dA G_d + A dG_d - i A G_d (dPhi - f dtau_d)),
// so the common phase factor cancels in Re(d_j r d_k r*): the Gram matrix
// needs no per-bin sincos, only the four intrinsic parameters (M_c, eta,
// chi1, chi2) are re-evaluated per bin (FP64), and the seven extrinsic ones
// reduce to per-request constants times three moments of A^2.  The
// per-bin products are FP32 with Kahan sums; assembly and the pivoted
// Cholesky inverse (util.cpp:857-900) are FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/gwgpu.h"
#include "capi_internal.h"
#include "fisher_ff.h"
#include "fisher_math.h"
#include "fisher_ref.h"
#include "kernel_util.cuh"
#include "kernels.h"

namespace gwf {
using namespace gwt;
using gwk::StreamDev;

constexpr int kBlock = 128;
constexpr int kStatusBounds = 0x100;  // set by a tile whose bins fall outside the tables
constexpr int kStatusRedo = 10;       // five-point source left to the reference algorithm (never returned)
constexpr int kStatusFp64 = 11;       // a source that two floats cannot hold, left to the FP64 sums (never returned)

// ------------------------------------------------------------- batched form
__global__ void k_fisher_slots(const GenParams *__restrict__ params, int nsrc, int method, const int *__restrict__ dets,
                               int ndet, double df, double epsilon, int step_mode, const double *__restrict__ qnm,
                               SlotOut *out) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nsrc * kSlots) return;
  fisher_slot(params[g / kSlots], g % kSlots, method, dets, ndet, df, epsilon, step_mode, qnm, out[g]);
}

// One warp per source: a lane per divisor, eight per waveform pair, then a lane
// per extrinsic row, and with FF the pairs' two-float coefficients the same way.
// Bound by the latency of a lane's FP64 chain; 256 sources x 3 detectors: 63
// us, one thread per source 292.
template <bool FF>
__global__ void __launch_bounds__(32) k_fisher_setup(const GenParams *__restrict__ params, int method, int ndet,
                                                     double epsilon, int step_mode, int order,
                                                     const SlotOut *__restrict__ slots, FisherSrc *out, FfSrc *ffout,
                                                     int *status, int *beyond) {
  const int src = blockIdx.x, lane = threadIdx.x;
  const unsigned all = 0xffffffffu;
  const SlotOut *S = slots + (size_t)src * kSlots;
  FisherSrc &F = out[src];
  // the waveforms: centre, + and - of the four pairs
  constexpr int kW = sizeof(WaveF64) / 4;
  static_assert(sizeof(WaveF64) % 4 == 0, "copied as words");
#pragma unroll
  for (int j = 0; j < 1 + 2 * kIntr; j++) {
    const unsigned *x = (const unsigned *)&S[j ? 14 + j : 0].w;
    unsigned *y = (unsigned *)(j == 0 ? &F.w0 : j & 1 ? &F.wp[j / 2] : &F.wm[j / 2 - 1]);
    for (int w = lane; w < kW; w += 32) y[w] = x[w];
  }
  const bool slot = lane < kSlots;
  const int st = (int)__reduce_or_sync(all, slot ? (unsigned)S[lane].status : 0u);
  const int cut = __reduce_max_sync(all, slot ? S[lane].w.n_cut : S[0].w.n_cut);
  if (lane == 0) {
    fisher_unpack(params[src], method, F.v, F.logf);
    F.status = status[src] = st;
    F.n_cut_any = cut;
  }
  __syncwarp();
  if (lane < kDim) fisher_setup_div(epsilon, step_mode, lane, F);
  __syncwarp();
  if (lane < kIntr) fisher_setup_rule(epsilon, step_mode, lane, F);
  __syncwarp();
  fisher_setup_pair(F.w0.A_scale, lane / 8, F, lane % 8, 8);
  for (int j = lane; j < ndet * (kCheap + 1); j += 32) {
    const int d = j / (kCheap + 1), i = j % (kCheap + 1);
    if (i < kCheap) fisher_setup_row(S, order, d, i, F);
    else fisher_setup_det(S, order, d, F);
  }
  __syncwarp();
  if (lane == 0) fisher_setup_route(order, F);
  if constexpr (FF) {
    FfSrc &X = ffout[src];
    bool ok = ff_pair(F, lane / 8, X.q[lane / 8], lane % 8, 8);
    if (lane == 1) ok = ff_centre(F, X) && ok;
    ok = __all_sync(all, ok);
    if (lane == 0) {
      X.ok = ok;
      if (!ok && !st && !F.needs_ref) *beyond = 1;
    }
  }
}

struct FisherArgs {
  const FisherSrc *src;
  int nsrc, ndet, nw;       // nw: distinct weight streams (1 when every detector has the same PSD)
  const int *wslot;         // detector -> weight stream
  const float *what[kMaxDet];
  double wscale[kMaxDet];
  // FP64 sums: the weight of bin k is c3 s_k / (S_k wscale) from the stream's
  // FP64 reciprocal PSD (Simpson pattern s_k, c3 = 4 df_s / 3), or iw_k / (S_k
  // wscale) for a stream registered with its own integration weights iw
  const double *ipsd[kMaxDet];
  const double *iw[kMaxDet];
  double c3[kMaxDet];
  int n0, N, tile, ntiles;
  double df, fisher_df_ratio;  // (f1 - f0) / simpson_df
  float df_f;                  // df in FP32 (the bins' frequency in the moment sums)
  gwt::Tables tab;
  const double *tm76d;
  int tm76d_n;              // tm76d valid for n <= tm76d_n
  // two-float sums: the sources' coefficients, the power tables, the weights
  const FfSrc *ff;
  gwt::AccTables acc;
  const gwt::AccLut *lut;
  const gwt::ff *wf[kMaxDet];
  unsigned *item_counter, *src_done;
  double *partials;  // items * kMaxDet * kSums
  double *fisher, *cov;
  const int *beyond;        // set: a source that two floats cannot hold is among them
  int *status;
};

// ACC64: the per-bin differences, weights and moment sums in FP64 instead of
// FP32 values with compensated FP32 sums.
template <int NW, bool ACC64>
__global__ void __launch_bounds__(kBlock, 3) k_fisher_main(const FisherArgs a) {
  __shared__ int s_item;
  __shared__ __align__(16) unsigned char s_buf[sizeof(FisherSrc)];
  __shared__ double s_red[32 * 8];
  const int tid = threadIdx.x;
  const int nitems = a.nsrc * a.ntiles;
  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(a.item_counter, 1u);
    __syncthreads();
    const int it = s_item;
    if (it >= nitems) break;
    const int src = it / a.ntiles, tile = it % a.ntiles;
    {
      const unsigned *p = (const unsigned *)(a.src + src);
      unsigned *q = (unsigned *)s_buf;
      for (int w = tid; w < (int)(sizeof(FisherSrc) / 4); w += blockDim.x) q[w] = p[w];
    }
    __syncthreads();
    const FisherSrc &F = *(const FisherSrc *)s_buf;
    using Acc = typename std::conditional<ACC64, double, KSum>::type;
    Acc acc[NW * kSums];
#pragma unroll
    for (int j = 0; j < NW * kSums; j++) {
      if constexpr (ACC64) acc[j] = 0.0;
      else acc[j] = KSum{0.f, 0.f};
    }
    const int k0 = tile * a.tile, k1 = min(k0 + a.tile, a.N);
    const bool in_tables = a.n0 >= 1 && a.n0 + k1 - 1 <= a.tab.nmax && a.n0 + k1 - 1 <= a.tm76d_n;
    if (!in_tables && tid == 0) atomicOr(a.status + src, kStatusBounds);
    if (F.status == 0 && in_tables) {
      for (int k = k0 + tid; k < k1; k += blockDim.x) {
        const int n = a.n0 + k;
        if constexpr (ACC64) {
          double a0, qr[kIntr], qi[kIntr];
          if (!fisher_bin_q(F, n, a.tab.t13[n], a.tab.tm53[n], a.tab.tln[n], a.tab.t34[n], a.tm76d[n],
                            a.tab.tm76f[n], a0, qr, qi))
            continue;
          const double fk = (double)n * a.df, sw = simpson_weight(k, a.N);
#pragma unroll
          for (int w = 0; w < NW; w++)
            fisher_accumulate64((a.iw[w] ? a.iw[w][k] : a.c3[w] * sw) * a.ipsd[w][k] / a.wscale[w], a0, fk, qr, qi,
                                acc + w * kSums);
        } else {
          float a0, qr[kIntr], qi[kIntr];
          if (!fisher_bin_q(F, n, a.tab.t13[n], a.tab.tm53[n], a.tab.tln[n], a.tab.t34[n], a.tm76d[n],
                            a.tab.tm76f[n], a0, qr, qi))
            continue;
          const float fk = (float)n * a.df_f;
#pragma unroll
          for (int w = 0; w < NW; w++) fisher_accumulate(a.what[w][k], a0, fk, qr, qi, acc + w * kSums);
        }
      }
    }
    // block reduction in FP64, 8 values at a time
    double *part = a.partials + (size_t)it * kMaxDet * kSums;
    for (int base = 0; base < NW * kSums; base += 8) {
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (base + j >= NW * kSums) v[j] = 0.0;
        else if constexpr (ACC64) v[j] = acc[base + j];
        else v[j] = (double)acc[base + j].s - (double)acc[base + j].c;
      }
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
      const int lane = tid & 31, warp = tid >> 5;
      if (lane == 0)
#pragma unroll
        for (int j = 0; j < 8; j++) s_red[warp * 8 + j] = v[j];
      __syncthreads();
      if (tid < 8 && base + tid < NW * kSums) {
        double s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += s_red[w * 8 + tid];
        part[base + tid] = s;
      }
      __syncthreads();
    }
    // last tile of this source: assemble Gamma in FP64 and invert
    __shared__ bool s_last;
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      unsigned prev = atomicAdd(a.src_done + src, 1u);
      s_last = (prev == (unsigned)a.ntiles - 1);
    }
    __syncthreads();
    // the source's sums over its tiles, one sum per thread in tile order
    __shared__ double s_sum[kMaxDet * kSums];
    if (s_last) {
      __threadfence();
      for (int j = tid; j < NW * kSums; j += blockDim.x) {
        double sj = 0;
        for (int tt = 0; tt < a.ntiles; tt++)
          sj += __ldcg(&a.partials[((size_t)(src * a.ntiles + tt)) * kMaxDet * kSums + j]);
        s_sum[j] = sj;
      }
    }
    __syncthreads();
    if (s_last && tid == 0) {
      const double *Ssum = s_sum;
      double Gm[kDim * kDim];
      fisher_assemble(F, Ssum, a.ndet, a.wslot, a.wscale, a.fisher_df_ratio, Gm);
      double *outF = a.fisher + (size_t)src * kDim * kDim;
      int st = F.status;
      if (__ldcg(a.status + src) & kStatusBounds) st = 5;
      for (int j = 0; j < kDim * kDim; j++) outF[j] = st ? __longlong_as_double(0x7ff8000000000000ll) : Gm[j];
      if (a.cov) {
        double inv[kDim * kDim];
        int cs = st ? 1 : chol_invert(Gm, inv, kDim);
        double *outC = a.cov + (size_t)src * kDim * kDim;
        for (int j = 0; j < kDim * kDim; j++) outC[j] = cs ? __longlong_as_double(0x7ff8000000000000ll) : inv[j];
        if (!st && cs) st = 9;  // inversion failed
      }
      if (!st && F.needs_ref) st = kStatusRedo;
      a.status[src] = st;
    }
    __syncthreads();
  }
}

// Sums 0..31 of v over the warp, in two floats: lane l is left with sum l.
__device__ __forceinline__ ff warp_sums(ff (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < o; j++) {
      const bool up = lane & o;
      const ff keep = up ? v[j + o] : v[j], send = up ? v[j] : v[j + o];
      v[j] = ff_norm(ff_add(keep, ff{__shfl_xor_sync(0xffffffffu, send.h, o), __shfl_xor_sync(0xffffffffu, send.l, o)}));
    }
  return v[0];
}
// A pair's difference in FP64 (bins that ff_pair_q leaves).
__device__ __noinline__ double2 pair_fp64(const FisherSrc *F, int q, int n, double t, double r, double lnn, double t34,
                                          double m76) {
  double2 v;
  fisher_pair_q<double>(*F, q, n, t, r, lnn, t34, m76, 0.f, wave64_amp(F->w0, n, t, m76), v.x, v.y);
  return v;
}

// The moment sums of the calls that take no inverse, in two floats.  An item is
// a tile of one source under one weight stream; a thread's sums run over
// kFfTile / kBlock terms, short enough for a two-float sum, the rest of the way
// up goes through one transposed warp sum and FP64.
// FP64 bins occupy the FP64 pipe for 64 cycles an instruction; here a bin is
// ~1,900 FP32 instructions (the differences of four pairs ~1,100, products and
// sums ~500), bound by their issue: 256 sources on 32,128 bins 5740 -> 560 us
// (745 with the four pairs' code unrolled at three blocks an SM).
// Where the inverse is wanted too the sums stay FP64: it magnifies them by the
// matrix's condition number.
constexpr int kFfTile = 2048;
__global__ void __launch_bounds__(kBlock, 4) k_fisher_ff(const __grid_constant__ FisherArgs a) {
  if (*a.beyond) return;  // the chunk takes FP64 sums
  __shared__ int s_item, s_last;
  __shared__ FfSrc S;
  __shared__ gwt::AccLut lut;
  __shared__ double s_red[kBlock / 32][32];
  __shared__ double s_sum[kMaxDet * kSums];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    const unsigned *p = (const unsigned *)a.lut;
    for (int w = tid; w < (int)(sizeof(gwt::AccLut) / 4); w += kBlock) ((unsigned *)&lut)[w] = p[w];
  }
  const int per = a.ntiles * a.nw, nitems = a.nsrc * per;
  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(a.item_counter, 1u);
    __syncthreads();
    const int it = s_item;
    if (it >= nitems) break;
    const int src = it / per, w = it % per / a.ntiles, tile = it % a.ntiles;
    const FisherSrc &F = a.src[src];
    const int k0 = tile * kFfTile;
    int k1 = min(k0 + kFfTile, a.N);
    const bool in_tables = a.n0 >= 1 && a.n0 + k1 - 1 <= a.tab.nmax && a.n0 + k1 - 1 <= a.tm76d_n &&
                           a.n0 + k1 - 1 <= a.acc.nmax;
    if (!in_tables && tid == 0) atomicOr(a.status + src, kStatusBounds);
    const bool run = F.status == 0 && !F.needs_ref && in_tables && a.ff[src].ok;
    k1 = run ? min(k1, F.n_cut_any - a.n0 + 1) : k0;
    double *part = a.partials + ((size_t)(src * a.ntiles + tile) * kMaxDet + w) * kSums;
    if (k0 < k1) {
      const unsigned *p = (const unsigned *)(a.ff + src);
      for (int j = tid; j < (int)(sizeof(FfSrc) / 4); j += kBlock) ((unsigned *)&S)[j] = p[j];
      __syncthreads();
      ff acc[32];
#pragma unroll
      for (int j = 0; j < 32; j++) acc[j] = ff{0.f, 0.f};
      for (int k = k0 + tid; k < k1; k += kBlock) {
        const int n = a.n0 + k;
        const FfBin b = ff_bin(a.acc, n);
        const ff a0 = ff_amp0(S, n, b, lut);
        ff qr[kIntr], qi[kIntr];
        // one copy of the pair's code: four of them exceed the instruction cache
#pragma unroll 1
        for (int q = 0; q < kIntr; q++) {
          ff vr, vi;
          if (!ff_pair_q(S.q[q], S.n_mid, n, b, lut, a0, vr, vi)) {
            const double2 v = pair_fp64(&F, q, n, a.tab.t13[n], a.tab.tm53[n], a.tab.tln[n], a.tab.t34[n], a.tm76d[n]);
            vr = ff_split(v.x);
            vi = ff_split(v.y);
          }
#pragma unroll
          for (int j = 0; j < kIntr; j++)
            if (j == q) {
              qr[j] = vr;
              qi[j] = vi;
            }
        }
        ff_accumulate(a.wf[w][k], a0, b.n, qr, qi, acc);
      }
      s_red[warp][lane] = ff_value(warp_sums(acc, lane));
      __syncthreads();
      if (tid < kSums) {
        double s = 0;
        for (int j = 0; j < kBlock / 32; j++) s += s_red[j][tid];
        part[tid] = s;
      }
    } else if (tid < kSums) {
      part[tid] = 0.0;
    }
    // the source's last tile adds the tiles in their order and assembles Gamma
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      s_last = atomicAdd(a.src_done + src, 1u) == (unsigned)per - 1;
    }
    __syncthreads();
    if (!s_last) continue;
    __threadfence();
    bool fin = a.ff[src].ok;
    for (int j = tid; j < a.nw * kSums; j += kBlock) {
      const int i = j % kSums;
      double s = 0;
      for (int t = 0; t < a.ntiles; t++)
        s += __ldcg(&a.partials[((size_t)(src * a.ntiles + t) * kMaxDet + j / kSums) * kSums + i]);
      if (!isfinite(s)) fin = false;
      if (i == 1 || (i >= 13 && ((i - 13) & 2))) s *= a.df;  // the bin number to its frequency
      if (i == 2) s *= a.df * a.df;
      s_sum[j] = s;
    }
    fin = __syncthreads_and(fin);
    int st = F.status;
    if (__ldcg(a.status + src) & kStatusBounds) st = 5;
    if (tid < kDim * (kDim + 1) / 2) {
      int i = 0, j = tid;
      while (j > i) j -= ++i;
      const double g = st ? __longlong_as_double(0x7ff8000000000000ll)
                          : fisher_element(F, s_sum, a.ndet, a.wslot, a.wscale, a.fisher_df_ratio, i, j);
      double *G = a.fisher + (size_t)src * kDim * kDim;
      G[i * kDim + j] = G[j * kDim + i] = g;
    }
    __syncthreads();
    if (tid == 0) a.status[src] = st ? st : (F.needs_ref ? kStatusRedo : (fin ? 0 : kStatusFp64));
  }
}

template <bool ACC64>
void launch_main(const FisherArgs &a, int nw, int grid, cudaStream_t s) {
  switch (nw) {
    case 1: k_fisher_main<1, ACC64><<<grid, kBlock, 0, s>>>(a); break;
    case 2: k_fisher_main<2, ACC64><<<grid, kBlock, 0, s>>>(a); break;
    case 3: k_fisher_main<3, ACC64><<<grid, kBlock, 0, s>>>(a); break;
    default: k_fisher_main<4, ACC64><<<grid, kBlock, 0, s>>>(a); break;
  }
}

// ---------------------------------------------------------------- plain form
// One parameter's central difference of the FP64 response (fisher.cpp:361-470).
struct FDReq {
  Request rp, rm, rpp, rmm;
};
__global__ void k_fisher_fd(const FDReq *__restrict__ fr, int order, int apply_shift, double div, double logscale,
                            const double *__restrict__ freqs, int N, double2 *__restrict__ deriv) {
  const FDReq &R = *fr;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
    double f = freqs[k];
    cd a, b, xp, xm;
    wave_bin(R.rp, f, a, b);
    xp = response_bin(R.rp.det[0], a, b, f, false);
    wave_bin(R.rm, f, a, b);
    xm = response_bin(R.rm.det[0], a, b, f, false);
    if (apply_shift) {  // exp(i (-2 pi DTOA) f) with DTOA from the perturbed sky position (:403-409)
      double s, c;
      sincos(R.rp.det[1].tau * f, &s, &c);
      xp = cmul(xp, cd{c, s});
      sincos(R.rm.det[1].tau * f, &s, &c);
      xm = cmul(xm, cd{c, s});
    }
    cd d;
    if (order >= 4) {  // five-point rule; the +-2 eps responses are time shifted, not phase shifted (:426-458)
      cd xpp, xmm;
      wave_bin(R.rpp, f, a, b);
      xpp = response_bin(R.rpp.det[0], a, b, f, false);
      wave_bin(R.rmm, f, a, b);
      xmm = response_bin(R.rmm.det[0], a, b, f, false);
      d.re = (-xpp.re + 8. * xp.re - 8. * xm.re + xmm.re) / div;
      d.im = (-xpp.im + 8. * xp.im - 8. * xm.im + xmm.im) / div;
    } else {
      d.re = (xp.re - xm.re) / div;
      d.im = (xp.im - xm.im) / div;
    }
    deriv[k] = make_double2(d.re * logscale, d.im * logscale);
  }
}

// Gram matrix 4 Simpson(Re(d_j d_k*)/S) (fisher.cpp:2704-2781), one block per (j, k).
__global__ void k_fisher_gram(const double2 *__restrict__ deriv, int dim, int N, const double *__restrict__ psd,
                              double df, double *out) {
  int j = blockIdx.x, k = blockIdx.y;
  if (k > j) return;
  const double2 *a = deriv + (size_t)j * N, *b = deriv + (size_t)k * N;
  double s = 0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    double w = simpson_weight(i, N);
    double2 x = a[i], y = b[i];
    s += w * ((x.x * y.x + x.y * y.y) / psd[i]);
  }
  __shared__ double sm[32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sm[w];
    double v = 4 * (t * df / 3);
    out[j * dim + k] = v;
    out[k * dim + j] = v;
  }
}

int det_index(const char *n) {
  static const char *names[9][3] = {{"Hanford", "hanford", ""},
                                    {"Livingston", "livingston", ""},
                                    {"Virgo", "virgo", ""},
                                    {"Kagra", "kagra", ""},
                                    {"Indigo", "indigo", ""},
                                    {"Cosmic Explorer", "cosmic explorer", "CE"},
                                    {"Einstein Telescope 1", "einstein telescope 1", "ET1"},
                                    {"Einstein Telescope 2", "einstein telescope 2", "ET2"},
                                    {"Einstein Telescope 3", "einstein telescope 3", "ET3"}};
  if (!n) return -1;
  for (int i = 0; i < 9; i++)
    for (int j = 0; j < 3; j++)
      if (names[i][j][0] && std::strcmp(n, names[i][j]) == 0) return i;
  return -1;
}

}  // namespace gwf

using namespace gwf;

extern "C" {

int gwgpu_fisher_numerical(gwgpu_context *c, const double *freqs, int N, const char *method, const char *detector,
                           const char *reference_detector, double *output, int dim, const gwgpu_gen_params *params,
                           int order, const double *noise) {
  if (!c || !freqs || N < 2 || !method || !output || !params || !noise) return GWGPU_EINVAL;
  std::string m(method);
  int meth = (m == "IMRPhenomD") ? 0 : (m == "MCMC_IMRPhenomD" ? 1 : -1);
  if (meth < 0 || dim != kDim || (order != 2 && order != 4)) return GWGPU_EINVAL;
  int det = det_index(detector), ref = det_index(reference_detector);
  if (det < 0 || ref < 0) return GWGPU_EINVAL;
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  GenParams in;
  std::memcpy(&in, params, sizeof(in));
  double v[kDim];
  int logf[kDim];
  fisher_unpack(in, meth, v, logf);
  const double epsilon = 1e-8;  // fisher.cpp:158
  size_t need = sizeof(double) * (size_t)N * (2 + 2 * (size_t)dim) + sizeof(double) * N + sizeof(FDReq) +
                sizeof(double) * dim * dim + 256;
  void *dev;
  int st = c->workspace(gwgpu_context::kWsFisher, need, &dev);
  if (st) return st;
  char *p = (char *)dev;
  double *df = (double *)p;
  p += sizeof(double) * N;
  double *dpsd = (double *)p;
  p += sizeof(double) * N;
  double2 *deriv = (double2 *)p;
  p += sizeof(double2) * (size_t)N * dim;
  double *dout = (double *)p;
  p += sizeof(double) * dim * dim;
  p = (char *)(((uintptr_t)p + 255) & ~(uintptr_t)255);
  FDReq *dreq = (FDReq *)p;
  cudaMemcpyAsync(df, freqs, sizeof(double) * N, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(dpsd, noise, sizeof(double) * N, cudaMemcpyHostToDevice, c->stream);
  FDReq *h;
  st = c->pinned(gwgpu_context::kHwsFisher, sizeof(FDReq) * dim, (void **)&h);
  if (st) return st;
  for (int i = 0; i < dim; i++) {
    double eps = epsilon, pv[kDim];
    GenParams q;
    double div = fisher_perturb(v, i, 1, eps, pv);
    fisher_repack(pv, in, meth, q);
    // det[0]: this detector's F+/Fx; det[1].tau: -2 pi DTOA(ref -> det) when ref != det
    int dd[2] = {det, ref};
    request_prologue(h[i].rp, q, kPhenomD, dd, 1, c->qnm_host.data());
    h[i].rp.det[1].tau = -2 * kPi * dtoa(q.RA, q.DEC, q.gmst, ref, det);
    fisher_perturb(v, i, -1, eps, pv);
    fisher_repack(pv, in, meth, q);
    request_prologue(h[i].rm, q, kPhenomD, dd, 1, c->qnm_host.data());
    h[i].rm.det[1].tau = -2 * kPi * dtoa(q.RA, q.DEC, q.gmst, ref, det);
    double d4 = div == eps ? 6. * eps : 12. * eps;
    if (order >= 4) {
      double pp[kDim];
      for (int j = 0; j < kDim; j++) pp[j] = v[j];
      bool onesided = (i == 8 && v[i] > .25 - eps);
      pp[i] = onesided ? v[i] : v[i] + 2 * eps;
      fisher_repack(pp, in, meth, q);
      if (ref != det) q.tc -= dtoa(q.RA, q.DEC, q.gmst, ref, det);
      request_prologue(h[i].rpp, q, kPhenomD, dd, 1, c->qnm_host.data());
      pp[i] = v[i] - 2 * eps;
      fisher_repack(pp, in, meth, q);
      if (ref != det) q.tc -= dtoa(q.RA, q.DEC, q.gmst, ref, det);
      request_prologue(h[i].rmm, q, kPhenomD, dd, 1, c->qnm_host.data());
    }
    double divisor = order >= 4 ? d4 : div;
    double logscale = logf[i] ? v[i] : 1.0;
    cudaMemcpyAsync(dreq, &h[i], sizeof(FDReq), cudaMemcpyHostToDevice, c->stream);
    int grid = (N + 127) / 128;
    k_fisher_fd<<<grid, 128, 0, c->stream>>>(dreq, order, ref != det, divisor, logscale, df, N, deriv + (size_t)i * N);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return c->fail(e, "fisher fd launch");
    e = cudaStreamSynchronize(c->stream);  // dreq is reused for the next parameter
    if (e != cudaSuccess) return c->fail(e, "fisher fd");
  }
  k_fisher_gram<<<dim3(dim, dim), 256, 0, c->stream>>>(deriv, dim, N, dpsd, freqs[1] - freqs[0], dout);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->fail(e, "fisher gram launch");
  cudaMemcpyAsync(output, dout, sizeof(double) * dim * dim, cudaMemcpyDeviceToHost, c->stream);
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->fail(e, "fisher");
  return GWGPU_OK;
}

}  // extern "C"

// The moment form for n sources; acc64 selects FP64 per-bin values and sums.
int gwf_moment_run(gwgpu_context *c, const gwgpu_gen_params *params, int n, int method, int order, const int *handles,
                   int ndet, double epsilon, int step_mode, double *fisher, double *covariance, int *status,
                   bool acc64) {
  if (!c || !params || n < 1 || !handles || ndet < 1 || ndet > kMaxDet || !fisher || (method != 0 && method != 1) ||
      (order != 2 && order != 4))
    return GWGPU_EINVAL;
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const gwgpu_context::Stream *s0 = c->get_stream(handles[0]);
  if (!s0) return GWGPU_ENOTFOUND;
  if (!s0->dev.uniform_int || s0->dev.iw) {
    c->last_error = "fisher_batch needs Simpson streams on a uniform grid with f0 a multiple of df";
    return GWGPU_EINVAL;
  }
  FisherArgs a;
  std::memset(&a, 0, sizeof(a));
  int dets[kMaxDet];
  std::vector<int> wslot(ndet);
  int nw = 0;
  std::vector<const gwgpu_context::Stream *> ws;
  for (int d = 0; d < ndet; d++) {
    const gwgpu_context::Stream *s = c->get_stream(handles[d]);
    if (!s) return GWGPU_ENOTFOUND;
    if (s->dev.N != s0->dev.N || s->dev.n0 != s0->dev.n0 || s->dev.iw) return GWGPU_EINVAL;
    dets[d] = s->dev.det;
    int found = -1;
    for (int w = 0; w < nw; w++) {  // same PSD and grid -> same weight stream
      if (ws[w]->dev.wscale == s->dev.wscale && ws[w]->psd_hash == s->psd_hash) {
        found = w;
        break;
      }
    }
    if (found < 0) {
      found = nw++;
      ws.push_back(s);
    }
    wslot[d] = found;
  }
  // the FP64 n^(-7/6) table
  int st = c->ensure_tm76d(s0->dev.n0 + s0->dev.N);
  if (st) return st;
  // Two-float sums for the FP64 calls without an inverse, on streams that have
  // their two-float weights and where there is memory for the sources' pairs.
  bool two_float = acc64 && !covariance;
  for (const auto *s : ws) two_float = two_float && s->dev.wf != nullptr;
  constexpr int kTile = 4096;  // of the FP64 and mixed sums: fewer tiles than kFfTile's
  const int N = s0->dev.N;
  const double df = s0->dev.df;
  // chunk sources to bound the scratch
  const int chunk = std::min(n, 2048);
  int ntiles;
  void *dev;
  for (;;) {
    const int tile = two_float ? kFfTile : kTile;
    ntiles = (N + tile - 1) / tile;
    const size_t bytes = sizeof(GenParams) * chunk + sizeof(SlotOut) * (size_t)chunk * kSlots + sizeof(FisherSrc) * chunk +
                         sizeof(double) * (size_t)chunk * ntiles * kMaxDet * kSums +
                         sizeof(double) * (size_t)chunk * 2 * kDim * kDim + sizeof(int) * (chunk + 8) +
                         sizeof(unsigned) * (chunk + 8) + sizeof(FfSrc) * (two_float ? chunk : 0) + 2048;
    st = c->workspace(gwgpu_context::kWsFisher + 10, bytes, &dev);
    if (!st) break;
    if (!two_float) return st;
    two_float = false;
  }
  auto align = [](char *p) { return (char *)(((uintptr_t)p + 255) & ~(uintptr_t)255); };
  char *p = (char *)dev;
  GenParams *dparams = (GenParams *)p;
  p = align(p + sizeof(GenParams) * chunk);
  SlotOut *slots = (SlotOut *)p;
  p = align(p + sizeof(SlotOut) * (size_t)chunk * kSlots);
  FisherSrc *srcs = (FisherSrc *)p;
  p = align(p + sizeof(FisherSrc) * chunk);
  double *partials = (double *)p;
  p = align(p + sizeof(double) * (size_t)chunk * ntiles * kMaxDet * kSums);
  double *dfish = (double *)p;
  p = align(p + sizeof(double) * (size_t)chunk * kDim * kDim);
  double *dcov = (double *)p;
  p = align(p + sizeof(double) * (size_t)chunk * kDim * kDim);
  int *dstat = (int *)p;
  p = align(p + sizeof(int) * (chunk + 8));
  unsigned *cnt = (unsigned *)p;
  p = align(p + sizeof(unsigned) * (chunk + 8));
  FfSrc *ffs = (FfSrc *)p;
  int *dwslot, *ddets;
  void *small;
  st = c->workspace(gwgpu_context::kWsFisher + 11, 256, &small);
  if (st) return st;
  dwslot = (int *)small;
  ddets = dwslot + kMaxDet;
  cudaMemcpyAsync(dwslot, wslot.data(), sizeof(int) * ndet, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(ddets, dets, sizeof(int) * ndet, cudaMemcpyHostToDevice, c->stream);
  a.ndet = ndet;
  a.nw = nw;
  a.wslot = dwslot;
  for (int w = 0; w < nw; w++) {
    a.what[w] = ws[w]->dev.what;
    a.wscale[w] = ws[w]->dev.wscale;
    a.ipsd[w] = ws[w]->dev.ipsd;
    a.iw[w] = ws[w]->dev.iw;
    a.c3[w] = 4. * ws[w]->dev.simpson_df / 3.;
    a.wf[w] = ws[w]->dev.wf;
  }
  a.ff = ffs;
  a.acc = c->acc;
  a.lut = c->acc_lut;
  a.n0 = s0->dev.n0;
  a.N = N;
  a.df = df;
  a.df_f = (float)df;
  a.fisher_df_ratio = (s0->host_freqs[1] - s0->host_freqs[0]) / s0->dev.simpson_df;
  a.tab = c->tables;
  a.tm76d = c->tm76d;
  a.tm76d_n = c->tm76d_n;
  static int grid_cache = 0, grid_ff = 0;
  if (!grid_cache) {
    cudaDeviceProp pr;
    cudaGetDeviceProperties(&pr, c->device);
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fisher_ff, kBlock, 0);
    grid_ff = pr.multiProcessorCount * std::max(per, 1);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fisher_main<1, false>, kBlock, 0);
    grid_cache = pr.multiProcessorCount * std::max(per, 1);
  }
  for (int s0i = 0; s0i < n; s0i += chunk) {
    int m = std::min(chunk, n - s0i);
    two_float = two_float && !c->two_float_off;  // its arrays may have given way to an allocation
    cudaMemcpyAsync(dparams, params + s0i, sizeof(GenParams) * m, cudaMemcpyHostToDevice, c->stream);
    int tot = m * kSlots;
    k_fisher_slots<<<(tot + 63) / 64, 64, 0, c->stream>>>(dparams, m, method, ddets, ndet, df, epsilon, step_mode,
                                                          c->qnm_dev, slots);
    cudaMemsetAsync(dstat + m, 0, sizeof(int), c->stream);
    if (two_float)
      k_fisher_setup<true><<<m, 32, 0, c->stream>>>(dparams, method, ndet, epsilon, step_mode, order, slots, srcs, ffs,
                                                    dstat, dstat + m);
    else
      k_fisher_setup<false><<<m, 32, 0, c->stream>>>(dparams, method, ndet, epsilon, step_mode, order, slots, srcs,
                                                     nullptr, dstat, nullptr);
    a.src = srcs;
    a.nsrc = m;
    a.item_counter = cnt + m;
    a.src_done = cnt;
    a.partials = partials;
    a.fisher = dfish;
    a.cov = covariance ? dcov : nullptr;
    a.status = dstat;
    a.beyond = dstat + m;
    std::vector<int> hs(m + 1);  // and the flag
    cudaError_t e = cudaSuccess;
    for (bool again = two_float;; again = false) {
      a.tile = again ? kFfTile : kTile;
      a.ntiles = (N + a.tile - 1) / a.tile;
      cudaMemsetAsync(cnt, 0, sizeof(unsigned) * (m + 8), c->stream);
      int grid = std::min(m * a.ntiles * (again ? nw : 1), again ? grid_ff : grid_cache);
      if (again) k_fisher_ff<<<grid, kBlock, 0, c->stream>>>(a);
      else if (acc64) launch_main<true>(a, nw, grid, c->stream);
      else launch_main<false>(a, nw, grid, c->stream);
      e = cudaGetLastError();
      if (e != cudaSuccess) return c->fail(e, "fisher batch launch");
      cudaMemcpyAsync(hs.data(), dstat, sizeof(int) * (m + 1), cudaMemcpyDeviceToHost, c->stream);
      cudaMemcpyAsync(fisher + (size_t)s0i * kDim * kDim, dfish, sizeof(double) * m * kDim * kDim,
                      cudaMemcpyDeviceToHost, c->stream);
      if (!again) break;
      e = cudaStreamSynchronize(c->stream);
      if (e != cudaSuccess) return c->fail(e, "fisher batch");
      // a source beyond what two floats hold, by its coefficients (nothing has run
      // then) or its sums: the chunk with FP64 sums
      if (!hs[m] && std::find(hs.begin(), hs.end() - 1, kStatusFp64) == hs.end() - 1) break;
    }
    if (covariance)
      cudaMemcpyAsync(covariance + (size_t)s0i * kDim * kDim, dcov, sizeof(double) * m * kDim * kDim,
                      cudaMemcpyDeviceToHost, c->stream);
    e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->fail(e, "fisher batch");
    // Sources whose matrix the sums leave indefinite (a normalised smallest
    // eigenvalue below their precision: ~1e-8 for the FP32-compensated sums,
    // near-equal masses and face-on orientations) are recomputed by the FP64
    // reference algorithm.
    std::vector<int> redo;
    for (int i = 0; i < m; i++)
      if (hs[i] == 9 || hs[i] == kStatusRedo) redo.push_back(i);
    if (!redo.empty()) {
      std::vector<GenParams> rp(redo.size());
      for (size_t j = 0; j < redo.size(); j++) std::memcpy(&rp[j], params + s0i + redo[j], sizeof(GenParams));
      std::vector<double> rf(redo.size() * kDim * kDim), rc(redo.size() * kDim * kDim);
      std::vector<int> rs(redo.size());
      st = gwf_ref_run(c, rp.data(), (int)redo.size(), method, order, handles, ndet, epsilon, step_mode, 0, rf.data(),
                       covariance ? rc.data() : nullptr, rs.data());
      if (st) return st;
      for (size_t j = 0; j < redo.size(); j++) {
        const size_t o = (size_t)(s0i + redo[j]) * kDim * kDim;
        std::memcpy(fisher + o, &rf[j * kDim * kDim], sizeof(double) * kDim * kDim);
        if (covariance) std::memcpy(covariance + o, &rc[j * kDim * kDim], sizeof(double) * kDim * kDim);
        hs[redo[j]] = rs[j];
      }
    }
    if (status)
      for (int i = 0; i < m; i++) status[s0i + i] = hs[i] == 9 ? GWGPU_ESINGULAR : gwk::status_code(hs[i]);
  }
  return GWGPU_OK;
}

extern "C" int gwgpu_fisher_batch(gwgpu_context *c, const gwgpu_gen_params *params, int n, int method,
                                  const int *handles, int ndet, double epsilon, int step_mode, double *fisher,
                                  double *covariance, int *status) {
  return gwf_moment_run(c, params, n, method, 2, handles, ndet, epsilon, step_mode, fisher, covariance, status, true);
}

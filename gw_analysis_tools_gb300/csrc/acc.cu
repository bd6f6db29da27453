// acc.cu -- the FP64 form on two-float bins (phenom_acc.h): the fused batch
// kernel, the one-request kernel, and the tables and stream pairs they read.
//
// Bound by FP32 issue: an IMRPhenomD bin with three detectors is ~550
// instructions, of which three sine/cosine pairs are 200, the ringdown phase
// and amplitude 200; per SM and second that leaves DRAM and L2 idle (a
// detector bin is 16 B of data and, once for shared weights, 8 B, from L2).
// Against the FP64 bins they took the place of (FP64 pipe full): 512
// IMRPhenomD requests on 3 x 32,128 bins 4,170 -> 256 us a call, 64
// IMRPhenomPv2 requests on 2 x 32,448 bins 973 -> 103 us, the one-request call
// on 3 x 32,128 bins 38.4 -> 22 us (Pv2, 3 x 16,224 bins: 48 -> 26 us), with
// an error against 80-bit references of 6e-13 instead of 9e-13 (Pv2 1e-13 instead
// of 3e-13; rms over 6 x 48 draws: t_c's turns leave no rounding behind).  512 requests on 3 x 3,000 quadrature nodes
// 745 -> 100 us (prologue 31): the powers of each node are tabulated
// at registration, its linear phases 128-bit products.
#include <cstdint>

#include "kernel_util.cuh"
#include "kernels.h"

namespace gwk {
using namespace gwt;

namespace {

// Blocks of 128 threads, five an SM (96 registers; a few spills from three detectors on): the reduction at an
// item's end then holds up a fifth of the SM's warps instead of half.  512
// IMRPhenomD requests on 3 x 32,128 bins: 250 us; two blocks of 256 threads 285,
// three 254, six of 128 255, ten of 64 265.
constexpr int kAccBlock = 128;
constexpr int kPlainBlock = 128;

__device__ __forceinline__ ff shfl_down_ff(ff v, int o) {
  return ff{__shfl_down_sync(0xffffffffu, v.h, o), __shfl_down_sync(0xffffffffu, v.l, o)};
}
// Sum over the warp (lane 0).
__device__ __forceinline__ ff warp_sum_ff(ff v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = ff_add(v, shfl_down_ff(v, o));
  return v;
}

// Bins k0, k0 + step, ... < k1 of one request into acc.
// (nodes: x's grid where it is not uniform; beyond the cut a node adds nothing).
template <int NDET, bool PV2>
__device__ __forceinline__ void acc_bins(const AccReq &x, const StreamDev *st, const AccTables &tb, const AccLut &lut,
                                         const AccNodes *nodes, int k0, int k1, int step, ff *acc) {
  const int n0 = st[0].n0;
  const bool wsh = x.m.wshared != 0;
  const float *dev = st[0].dev;
  for (int k = k0; k < k1; k += step) {
    ff4 wd[NDET];
    ff w[NDET];
#pragma unroll
    for (int d = 0; d < NDET; d++) {
      wd[d] = acc_ld(st[d].wd + k);
      if (d == 0 || !wsh) {
        const float2 v = __ldg((const float2 *)st[d].wf + k);
        w[d] = ff{v.x, v.y};
      }
    }
    if (nodes) {
      const int64_t f = __ldg((const long long *)st[0].freqs + k);
      if (f > x.fcut) continue;
      acc[0].h += x.bad;  // a phase that is not a number, where a node is live
      const float2 v = __ldg((const float2 *)nodes->x + k);
      const AccNode b{k, f, __ldg((const long long *)nodes->X + k), ff{v.x, v.y}, 0};
      if constexpr (PV2) acc_bin_p<NDET>(x, b, nodes->tb, lut, wd, w, wsh, acc);
      else acc_bin_d<NDET>(x, b, nodes->tb, lut, wd, w, wsh, acc);
      continue;
    }
    const AccBin b{n0 + k, dev ? acc_dev_turns(x, __ldg(dev + k)) : 0};
    if constexpr (PV2) acc_bin_p<NDET>(x, b, tb, lut, wd, w, wsh, acc);
    else acc_bin_d<NDET>(x, b, tb, lut, wd, w, wsh, acc);
  }
}

// The block's share of log L: its sums times the request's factors.  Warps
// reduce in two floats, thread 0 adds the warps in FP64 in order.  s_red: one
// double per warp.  bad: x.bad where the block has live bins.  Valid in thread 0.
template <int NDET, bool PV2>
__device__ __forceinline__ double acc_reduce(const AccReq &x, const ff *acc, double bad, double *s_red) {
  constexpr int NA = PV2 ? kAccPerDet : 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double v = 0.0;
#pragma unroll
  for (int d = 0; d < NDET; d++)
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const double t = ff_value(warp_sum_ff(acc[d * NA + j]));
      if (lane == 0 && t != 0.0) v += x.m.fc[d * kAccPerDet + j] * t;  // an infinite factor: only with bins
    }
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  double r = bad;
  if (threadIdx.x == 0)
    for (int w = 0; w < nw; w++) r += s_red[w];
  return r;
}
// Bins k0, k0 + blockDim.x .. below kend on the whole block; the result in thread 0.
template <int NDET>
__device__ __forceinline__ double acc_block(const AccReq &x, const StreamDev *st, const AccTables &tb,
                                            const AccLut &lut, const AccNodes *nodes, int k0, int kend,
                                            double *s_red) {
  // the model is zero beyond the cut
  const int kcut = nodes ? kend : min(kend, x.m.n_cut - st[0].n0 + 1);
  const double bad = !nodes && kcut > k0 ? x.bad : 0.f;
  if (x.m.approximant == kPhenomPv2) {
    ff acc[NDET * kAccPerDet];
#pragma unroll
    for (int j = 0; j < NDET * kAccPerDet; j++) acc[j] = ff{0.f, 0.f};
    acc_bins<NDET, true>(x, st, tb, lut, nodes, k0 + threadIdx.x, kcut, blockDim.x, acc);
    return acc_reduce<NDET, true>(x, acc, bad, s_red);
  }
  ff acc[NDET * 2];
#pragma unroll
  for (int j = 0; j < NDET * 2; j++) acc[j] = ff{0.f, 0.f};
  acc_bins<NDET, false>(x, st, tb, lut, nodes, k0 + threadIdx.x, kcut, blockDim.x, acc);
  return acc_reduce<NDET, false>(x, acc, bad, s_red);
}

__device__ __forceinline__ void copy_words(void *dst, const void *src, int bytes) {
  for (int w = threadIdx.x; w < bytes / 4; w += blockDim.x) ((unsigned *)dst)[w] = __ldcg((const unsigned *)src + w);
}

// ------------------------------------------------------------------- batch
// Persistent over the items in work order (as k_batch): an item is a tile of
// one request's bins, its partial sum one double; a warp of the block that finishes
// a request's last item adds them in a fixed order.  NODES: some requests' grids are
// not uniform (a kernel of its own, so that batches without them keep their
// code small).
template <int NDET, bool NODES>
__global__ void __launch_bounds__(kAccBlock, 5) k_batch_acc(const BatchArgs a) {
  __shared__ AccLut lut;
  __shared__ __align__(16) unsigned char s_req[sizeof(AccReq)];
  __shared__ StreamDev s_st[NDET];
  __shared__ AccNodes s_nodes;
  __shared__ double s_red[kAccBlock / 32];
  __shared__ int s_item, s_iid, s_bstart[kOrderBuckets + 1];
  const int tid = threadIdx.x;
  copy_words(&lut, a.lut, sizeof(AccLut));
  grid_dep_wait();  // the prologue's output
  if (a.bucket_fill && tid < 32) order_starts(a, s_bstart);
  __syncthreads();
  for (;;) {
    if (tid == 0) {
      const int it = (int)atomicAdd(a.item_counter, 1u);
      s_item = it;
      s_iid = order_item(a, s_bstart, it);
    }
    __syncthreads();
    if (s_item >= (a.bucket_fill ? s_bstart[kOrderBuckets] : a.nitems)) break;
    const int iid = s_iid;
    const Item I = a.items[iid];
    static_assert(sizeof(AccReq) % 4 == 0, "copied as words");
    copy_words(s_req, a.areq + I.req, sizeof(AccReq));
    if (tid < NDET) {
      StreamDev s = a.streams[__ldcg(a.handles + I.req * a.ndet + tid)];
      if (NODES && s.node) {
        s.wd = s.node->wd;
        s.wf = s.node->wf;
        if (tid == 0) s_nodes = *s.node;
      }
      s_st[tid] = s;
    }
    __syncthreads();
    const AccReq &x = *(const AccReq *)s_req;
    const int kend = min(I.k0 + a.tile, s_st[0].N);
    double v = 0.0;
    if (x.m.status == 0) v = acc_block<NDET>(x, s_st, a.acc, lut, NODES && s_st[0].node ? &s_nodes : nullptr, I.k0, kend, s_red);
    if (tid == 0) a.partials[iid] = v;
    if (arrive_last(a.req_done + I.req, (unsigned)__ldcg(a.item_count + I.req)) && tid < 32) {
      const int i0 = __ldcg(a.item_start + I.req), ic = __ldcg(a.item_count + I.req), st = x.m.status;
      double ll = 0.0;
      for (int q = tid; q < ic; q += 32) ll += __ldcg(a.partials + i0 + q);
      ll = warp_sum(ll);
      if (tid == 0) {
        a.out[I.req] = st ? __longlong_as_double(0x7ff8000000000000ll) : ll;
        a.status_out[I.req] = st;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------- plain
struct PlainAccStreams {
  StreamDev s[kMaxDet];
};
// One bin per thread; the last block adds the blocks' sums.  NODES: the grid's
// node arrays instead of the bins (beyond the cut a node adds nothing).
template <int NDET, bool NODES>
__global__ void __launch_bounds__(kPlainBlock) k_plain_acc(const __grid_constant__ AccReq x,
                                                           const __grid_constant__ PlainAccStreams ps,
                                                           const __grid_constant__ AccTables tb,
                                                           const AccLut *__restrict__ glut, double *partials,
                                                           unsigned *counter, double *out) {
  __shared__ AccLut lut;
  __shared__ double s_red[kPlainBlock / 32];
  __shared__ StreamDev s_st[NODES ? NDET : 1];
  __shared__ AccNodes s_nodes;
  const int tid = threadIdx.x, N = ps.s[0].N, k0 = blockIdx.x * kPlainBlock;
  double v = 0.0;
  if (NODES || k0 < x.m.n_cut - ps.s[0].n0 + 1) {
    copy_words(&lut, glut, sizeof(AccLut));
    if (NODES && tid < NDET) {
      StreamDev s = ps.s[tid];
      s.wd = s.node->wd;
      s.wf = s.node->wf;
      if (tid == 0) s_nodes = *s.node;
      s_st[tid] = s;
    }
    __syncthreads();
    v = acc_block<NDET>(x, NODES ? s_st : ps.s, tb, lut, NODES ? &s_nodes : nullptr, k0, min(k0 + kPlainBlock, N), s_red);
  }
  if (tid == 0) partials[blockIdx.x] = v;
  if (arrive_last(counter, gridDim.x)) {
    double t = 0.0;
    for (unsigned b = tid; b < gridDim.x; b += kPlainBlock) t += __ldcg(partials + b);
    t = warp_sum(t);
    __syncthreads();
    if ((tid & 31) == 0) s_red[tid >> 5] = t;
    __syncthreads();
    if (tid == 0) {
      double ll = 0.0;
      for (int w = 0; w < kPlainBlock / 32; w++) ll += s_red[w];
      out[0] = ll;
      *counter = 0;
    }
  }
}

// ------------------------------------------------------------------ tables
__device__ __forceinline__ ff4 two_pairs(double a, double b) {
  const ff u = ff_split(a), v = ff_split(b);
  return ff4{u.h, u.l, v.h, v.l};
}
__global__ void k_acc_tables(const AccTables tb) {
  for (int n = 1 + blockIdx.x * blockDim.x + threadIdx.x; n <= tb.nmax; n += gridDim.x * blockDim.x) {
    const double x = (double)n, t = tb.t13[n];
    const_cast<ff4 *>(tb.pw)[n] = two_pairs(t, pow_m7_6(x));
    const_cast<ff4 *>(tb.ph)[n] = two_pairs(1.0 / x, tb.t34[n]);
    const_cast<ff4 *>(tb.pv)[n] = two_pairs(1.0 / t, tb.tln[n]);
  }
}
// W_k = weight_k / S_k (register_stream's whitening), as pairs.
__global__ void k_acc_stream(const StreamDev d, int with_dev) {
  const double c3 = 4. * d.simpson_df / 3.;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.N; k += gridDim.x * blockDim.x) {
    const double W = (d.iw ? d.iw[k] : c3 * simpson_weight(k, d.N)) / d.psd[k];
    const double2 v = ((const double2 *)d.data)[k];
    const_cast<ff4 *>(d.wd)[k] = two_pairs(W * v.x / d.dscale, W * v.y / d.dscale);
    const_cast<ff *>(d.wf)[k] = ff_split(W / d.wscale);
    if (with_dev) const_cast<float *>(d.dev)[k] = (float)fma(-(double)(d.n0 + k), d.dfq, d.freqs[k]);
  }
}

// The same for a grid of nodes.
__global__ void k_acc_nodes(const StreamDev d, const AccNodes a) {
  const double idf = 1.0 / d.dfq;  // a power of two
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.N; k += gridDim.x * blockDim.x) {
    const double x = d.freqs[k] * idf, t = cbrt(x), ln = log(x), q = sqrt(x * sqrt(x));
    const_cast<ff4 *>(a.tb.pw)[k] = two_pairs(t, pow_m7_6(x));
    const_cast<ff4 *>(a.tb.ph)[k] = two_pairs(1.0 / x, q);
    const_cast<ff4 *>(a.tb.pv)[k] = two_pairs(1.0 / t, ln);
    const_cast<double *>(a.tb.t13)[k] = t;
    const_cast<double *>(a.tb.tm53)[k] = 1.0 / (x * (t * t));
    const_cast<double *>(a.tb.tln)[k] = ln;
    const_cast<double *>(a.tb.t34)[k] = q;
    const_cast<int64_t *>(a.X)[k] = (int64_t)llrint(x * 4398046511104.0);  // 2^kNodeBits
    const_cast<ff *>(a.x)[k] = ff_split(x);
  }
}

const void *acc_fn(int ndet, bool nodes) {
  switch (ndet + (nodes ? kMaxDet : 0)) {
    case 1: return (const void *)k_batch_acc<1, false>;
    case 2: return (const void *)k_batch_acc<2, false>;
    case 3: return (const void *)k_batch_acc<3, false>;
    case 4: return (const void *)k_batch_acc<4, false>;
    case kMaxDet + 1: return (const void *)k_batch_acc<1, true>;
    case kMaxDet + 2: return (const void *)k_batch_acc<2, true>;
    case kMaxDet + 3: return (const void *)k_batch_acc<3, true>;
    case kMaxDet + 4: return (const void *)k_batch_acc<4, true>;
    default: return nullptr;
  }
}

}  // namespace

int batch_acc_occupancy(int ndet, bool nodes) {
  int nb = 0;
  const void *f = acc_fn(ndet, nodes);
  if (!f || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, kAccBlock, 0) != cudaSuccess) return 1;
  return nb;
}
cudaError_t launch_batch_acc(const BatchArgs &a, bool nodes, int grid, cudaStream_t s, bool pdl) {
  const void *f = acc_fn(a.ndet, nodes);
  if (!f) return cudaErrorInvalidValue;
  void *args[] = {(void *)&a};
  return launch_dependent(f, dim3(grid), dim3(kAccBlock), args, s, pdl);
}
template <int NDET>
static void launch_plain_acc(const AccReq &x, const PlainAccStreams &ps, bool nodes, const AccTables &tab,
                             const AccLut *lut, double *partials, unsigned *counter, double *out, cudaStream_t s) {
  const int grid = plain_blocks(ps.s[0].N);
  if (nodes) k_plain_acc<NDET, true><<<grid, kPlainBlock, 0, s>>>(x, ps, tab, lut, partials, counter, out);
  else k_plain_acc<NDET, false><<<grid, kPlainBlock, 0, s>>>(x, ps, tab, lut, partials, counter, out);
}
cudaError_t launch_plain_acc(const AccReq &x, const StreamDev *streams, int ndet, const AccTables &tab,
                             const AccLut *lut, double *partials, unsigned *counter, double *out, cudaStream_t s) {
  PlainAccStreams ps;
  for (int d = 0; d < ndet; d++) ps.s[d] = streams[d];
  const bool nodes = streams[0].node != nullptr;
  switch (ndet) {
    case 1: launch_plain_acc<1>(x, ps, nodes, tab, lut, partials, counter, out, s); break;
    case 2: launch_plain_acc<2>(x, ps, nodes, tab, lut, partials, counter, out, s); break;
    case 3: launch_plain_acc<3>(x, ps, nodes, tab, lut, partials, counter, out, s); break;
    case 4: launch_plain_acc<4>(x, ps, nodes, tab, lut, partials, counter, out, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
bool plain_two_float(const Request &r, const StreamDev *streams, int ndet, const AccTables &tab, const AccLut *lut) {
  bool bins = lut && !r.m.status && streams[0].n0 + streams[0].N - 1 <= tab.nmax, nodes = lut && !r.m.status;
  for (int d = 0; d < ndet; d++) {
    bins = bins && streams[d].wd;
    nodes = nodes && streams[d].node;
  }
  return bins || nodes;
}
cudaError_t launch_plain_any(const Request &r, const FastX &fx, const StreamDev *streams, int ndet,
                             const AccTables &tab, const AccLut *lut, double *partials, unsigned *counter, double *out,
                             cudaStream_t s) {
  if (!plain_two_float(r, streams, ndet, tab, lut)) return launch_plain(r, streams, ndet, partials, counter, out, nullptr, s);
  double ds[kMaxDet], ws[kMaxDet];
  unsigned long long wk[kMaxDet];
  for (int d = 0; d < ndet; d++) {
    ds[d] = streams[d].dscale;
    ws[d] = streams[d].wscale;
    wk[d] = streams[d].wkey;
  }
  AccReq x;
  fast_acc(r, fx, grid_const(streams[0].dfq), x, ds, ws, wk);
  if (streams[0].node) acc_node_coeffs(r, streams[0].dfq, x);
  return launch_plain_acc(x, streams, ndet, tab, lut, partials, counter, out, s);
}
template <int NDET>
static cudaError_t plain_acc_preload_n() {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, k_plain_acc<NDET, false>);
  return e == cudaSuccess ? cudaFuncGetAttributes(&a, k_plain_acc<NDET, true>) : e;
}
cudaError_t plain_acc_preload() {
  cudaError_t e = plain_acc_preload_n<1>();
  if (e == cudaSuccess) e = plain_acc_preload_n<2>();
  if (e == cudaSuccess) e = plain_acc_preload_n<3>();
  if (e == cudaSuccess) e = plain_acc_preload_n<4>();
  return e;
}
cudaError_t launch_acc_tables(const AccTables &tab, cudaStream_t s) {
  k_acc_tables<<<(tab.nmax + 255) / 256, 256, 0, s>>>(tab);
  return cudaGetLastError();
}
cudaError_t launch_acc_nodes(const StreamDev &d, const AccNodes &a, cudaStream_t s) {
  StreamDev t = d;
  t.wd = a.wd;
  t.wf = a.wf;
  k_acc_nodes<<<(d.N + 255) / 256, 256, 0, s>>>(d, a);
  k_acc_stream<<<(d.N + 255) / 256, 256, 0, s>>>(t, 0);
  return cudaGetLastError();
}
cudaError_t launch_acc_stream(const StreamDev &d, bool with_dev, cudaStream_t s) {
  k_acc_stream<<<(d.N + 255) / 256, 256, 0, s>>>(d, with_dev ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace gwk

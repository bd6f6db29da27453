// conv.cu -- the Bluestein convolution of the maximised likelihood's FP32
// search: rows of N samples, zero-padded to M = M1 M2 (a power of two), in place.
//
// The length-M transform is split as j = j1 M2 + j2, k = k1 + M1 k2:
//   columns  transform over j1 for each j2, times w_M^{j2 k1}
//   rows     for each k1: transform over j2, times the chirp's spectrum, and the
//            inverse transform over k2 straight from registers
//   back     times w_M^{-j2 k1}, inverse transform over k1
// so that the forward and inverse transforms and the product take three passes
// over memory instead of five, the output is in order, and the zero half is
// neither read nor (at the end) written.  Bound by memory: 8 B read and written
// per entry and pass (half of it in the first and last); 384 rows of 32,128 samples,
// M = 2^16: 65 + 79 + 57 us, the two library transforms and the product between
// them 434 us.  Splitting the rows into groups that L2 holds between the passes
// costs more in launches and part-filled ends than it saves (668 -> 721 us for
// the call at 48 MB); moduli in rows of their own instead of in place lose the lines
// that L2 still holds (last pass 57 -> 94 us).
//
// A thread keeps 16 samples in registers between the passes of a transform
// (radix 16, then 2, 4, 8 or 16; samples u + m L / 16 at every boundary), a block
// 4,096 in shared memory for the exchanges: 16 columns of 256 samples are whole
// 128 B lines.  Three blocks an SM (80 registers) for the loads in flight; the
// last pass holds its twiddles beside the samples and takes two.
#include "conv.h"

namespace gwk {
namespace {

constexpr int kThreads = 256, kPoints = 16 * kThreads, kTab = 512;

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
template <bool INV>  // a w, or a conj(w)
__device__ __forceinline__ float2 twid(float2 a, float2 w) {
  if (INV) w.y = -w.y;
  return make_float2(fmaf(a.x, w.x, -(a.y * w.y)), fmaf(a.x, w.y, a.y * w.x));
}
template <bool INV>  // a times w_4
__device__ __forceinline__ float2 turn(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d) {
  const float2 s = cadd(a, c), t = csub(a, c), p = cadd(b, d), q = turn<INV>(csub(b, d));
  a = cadd(s, p);
  b = cadd(t, q);
  c = csub(s, p);
  d = csub(t, q);
}
// t[r] -> sum_r t[r] w_R^{r k}
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 *t) {
  if constexpr (R == 2) {
    const float2 a = t[0];
    t[0] = cadd(a, t[1]);
    t[1] = csub(a, t[1]);
  } else if constexpr (R == 4) {
    dft4<INV>(t[0], t[1], t[2], t[3]);
  } else {  // r = (R / 4) a + b, k = c + 4 d
    constexpr int B = R / 4;
    constexpr float kC[8] = {1.f, 0.923879532511287f, 0.707106781186548f, 0.382683432365090f, 0.f,
                             -0.382683432365090f, -0.707106781186548f, -0.923879532511287f};
    constexpr float kS[8] = {0.f, -0.382683432365090f, -0.707106781186548f, -0.923879532511287f, -1.f,
                             -0.923879532511287f, -0.707106781186548f, -0.382683432365090f};
#pragma unroll
    for (int b = 0; b < B; b++) {
      dft4<INV>(t[b], t[B + b], t[2 * B + b], t[3 * B + b]);  // c at c B + b
#pragma unroll
      for (int c = 1; c < 4; c++) {
        constexpr int kStep = 16 / R;
        const int e = b * c * kStep;  // w_16^e, e <= 9
        if (e == 0) continue;
        const float2 w = e < 8 ? make_float2(kC[e], kS[e]) : make_float2(-kC[e - 8], -kS[e - 8]);
        t[c * B + b] = twid<INV>(t[c * B + b], w);
      }
    }
    float2 o[R];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      float2 y[B];
#pragma unroll
      for (int b = 0; b < B; b++) y[b] = t[c * B + b];
      dft<B, INV>(y);
#pragma unroll
      for (int d = 0; d < B; d++) o[c + 4 * d] = y[d];
    }
#pragma unroll
    for (int k = 0; k < R; k++) t[k] = o[k];
  }
}
// One pass of radix R after passes whose radices multiply to NS.  at(i): sample
// i's place in the block's exchange buffer.
template <int L, int R, int NS, bool INV, class At>
__device__ __forceinline__ void pass(float2 (&v)[16], int u, const float2 *tab, float2 *s, At at) {
  constexpr int NB = 16 / R;
  constexpr bool last = R * NS == L;
  if (!last) __syncthreads();  // the buffer's last reads
#pragma unroll
  for (int b = 0; b < NB; b++) {
    float2 t[R];
#pragma unroll
    for (int r = 0; r < R; r++) t[r] = v[b + r * NB];
    const int j = u + b * (L / 16), k = j & (NS - 1);
    if (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) t[r] = twid<INV>(t[r], tab[NS == 16 ? r * 16 + k : 256 + k]);
    }
    dft<R, INV>(t);
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (last) v[b + r * NB] = t[r];
      else s[at((j - k) * R + k + r * NS)] = t[r];
    }
  }
  if (!last) {
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; m++) v[m] = s[at(u + m * (L / 16))];
  }
}
// The length-L transform of samples u + m L / 16, m = 0..15, of each thread.
template <int L, bool INV, class At>
__device__ __forceinline__ void transform(float2 (&v)[16], int u, const float2 *tab, float2 *s, At at) {
  pass<L, 16, 1, INV>(v, u, tab, s, at);
  constexpr int R = L / 16 < 16 ? L / 16 : 16;
  pass<L, R, 16, INV>(v, u, tab, s, at);
  if constexpr (L > 256) pass<L, L / 256, 256, INV>(v, u, tab, s, at);
}

// w_{16 R}^{r k} at r * 16 + k for the second pass (R = L / 16, at most 16), w_512^k
// at 256 + k for the third: lanes with neighbouring k read neighbouring places.
template <int L>
__device__ __forceinline__ void load_tab(float2 *s_tab, const float2 *tab) {
  constexpr int R = L / 16 < 16 ? L / 16 : 16;
  const int r = threadIdx.x / 16, k = threadIdx.x % 16;
  if (r < R) s_tab[threadIdx.x] = tab[r * k * (kTab / (16 * R))];
  if (L > 256) s_tab[256 + threadIdx.x] = tab[threadIdx.x];
  __syncthreads();
}

// Columns: INV = false the first step, true the last.
template <int L, bool INV>
__global__ void __launch_bounds__(kThreads, INV ? 2 : 3) k_conv_cols(float2 *__restrict__ a, int rows, int N, int M2,
                                                        const float2 *__restrict__ tw, const float2 *__restrict__ tab) {
  constexpr int C = kPoints / L;
  __shared__ float2 s[kPoints], s_tab[L > 256 ? 512 : 256];
  load_tab<L>(s_tab, tab);
  const int c = threadIdx.x % C, u = threadIdx.x / C, col = blockIdx.x * C + c;
  auto at = [&](int i) { return i * C + c; };
  for (int row = blockIdx.y; row < rows; row += gridDim.y) {
    float2 *x = a + (size_t)row * L * M2;
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int i = (u + m * (L / 16)) * M2 + col;
      if (INV) v[m] = twid<true>(x[i], __ldg(tw + i));
      else v[m] = i < N ? x[i] : make_float2(0.f, 0.f);
    }
    transform<L, INV>(v, u, s_tab, s, at);
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int i = (u + m * (L / 16)) * M2 + col;
      if (!INV) x[i] = twid<false>(v[m], __ldg(tw + i));
      else if (i < N) x[i] = v[m];
    }
  }
}
// Rows: forward, the chirp's spectrum, inverse.
template <int L>
__global__ void __launch_bounds__(kThreads, 3) k_conv_rows(float2 *__restrict__ a, int rows, int M,
                                                        const float2 *__restrict__ spec,
                                                        const float2 *__restrict__ tab) {
  constexpr int C = kPoints / L, U = L / 16;
  __shared__ float2 s[kPoints + kPoints / 16], s_tab[L > 256 ? 512 : 256];  // a place in 16 left free: no bank conflicts
  load_tab<L>(s_tab, tab);
  const int u = threadIdx.x % U, c = threadIdx.x / U, base = (blockIdx.x * C + c) * L;
  auto at = [&](int i) { return c * (L + L / 16) + i + i / 16; };
  for (int row = blockIdx.y; row < rows; row += gridDim.y) {
    float2 *x = a + (size_t)row * M + base;
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; m++) v[m] = x[u + m * U];
    transform<L, false>(v, u, s_tab, s, at);
#pragma unroll
    for (int m = 0; m < 16; m++) v[m] = twid<false>(v[m], __ldg(spec + base + u + m * U));
    transform<L, true>(v, u, s_tab, s, at);
#pragma unroll
    for (int m = 0; m < 16; m++) x[u + m * U] = v[m];
  }
}

__global__ void k_conv_tables(const float2 *__restrict__ B, int M1, int M2, float2 *__restrict__ tw,
                              float2 *__restrict__ spec, float2 *__restrict__ tab) {
  const int M = M1 * M2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    const int k1 = i / M2, j = i % M2;
    double sn, cs;
    sincospi(-2.0 * (double)(k1 * j) / (double)M, &sn, &cs);
    tw[i] = make_float2((float)cs, (float)sn);
    spec[i] = B[k1 + M1 * j];
    if (i < kTab) {
      sincospi(-2.0 * (double)i / (double)kTab, &sn, &cs);
      tab[i] = make_float2((float)cs, (float)sn);
    }
  }
}

// M1 >= M2, each of 128..512.  Shorter rows fit one block of a library transform,
// two launches instead of three: 24 and 384 rows of 2^13 take 2 us more and 2 us
// less here, of 2^14 4 and 25 us less (calls of 181 and 285 us).
bool split(int M, int *M1, int *M2) {
  if (M < 16384 || M > 512 * 512 || (M & (M - 1))) return false;
  int m = 0;
  while ((1 << m) < M) m++;
  *M1 = 1 << ((m + 1) / 2);
  *M2 = M / *M1;
  return true;
}
template <int L>
void cols(bool inv, float2 *a, int rows, int N, int M2, const ConvTables &t, cudaStream_t s) {
  const dim3 grid(M2 / (kPoints / L), rows < 2048 ? (rows + 1) / 2 : 1024);
  if (inv) k_conv_cols<L, true><<<grid, kThreads, 0, s>>>(a, rows, N, M2, t.tw, t.tab);
  else k_conv_cols<L, false><<<grid, kThreads, 0, s>>>(a, rows, N, M2, t.tw, t.tab);
}
void cols_any(int L, bool inv, float2 *a, int rows, int N, int M2, const ConvTables &t, cudaStream_t s) {
  if (L == 128) cols<128>(inv, a, rows, N, M2, t, s);
  else if (L == 256) cols<256>(inv, a, rows, N, M2, t, s);
  else cols<512>(inv, a, rows, N, M2, t, s);
}
template <int L>
void mid(float2 *a, int rows, int M, const ConvTables &t, cudaStream_t s) {
  const dim3 grid(M / kPoints, rows < 2048 ? (rows + 1) / 2 : 1024);
  k_conv_rows<L><<<grid, kThreads, 0, s>>>(a, rows, M, t.spec, t.tab);
}

}  // namespace

size_t conv_table_bytes(int M) {
  int a, b;
  return split(M, &a, &b) ? sizeof(float2) * (2 * (size_t)M + kTab) : 0;
}
ConvTables conv_tables_at(void *p, int M) {
  float2 *f = (float2 *)p;
  return ConvTables{f, f + M, f + 2 * (size_t)M};
}
cudaError_t launch_conv_tables(const float2 *B, int M, void *p, cudaStream_t s) {
  int a, b;
  if (!split(M, &a, &b)) return cudaErrorInvalidValue;
  const ConvTables t = conv_tables_at(p, M);
  k_conv_tables<<<(M + 255) / 256, 256, 0, s>>>(B, a, b, (float2 *)t.tw, (float2 *)t.spec, (float2 *)t.tab);
  return cudaGetLastError();
}
cudaError_t launch_conv(float2 *a, int rows, int N, int M, const ConvTables &t, cudaStream_t s) {
  int M1, M2;
  if (!split(M, &M1, &M2)) return cudaErrorInvalidValue;
  cols_any(M1, false, a, rows, N, M2, t, s);
  if (M2 == 128) mid<128>(a, rows, M, t, s);
  else if (M2 == 256) mid<256>(a, rows, M, t, s);
  else mid<512>(a, rows, M, t, s);
  cols_any(M1, true, a, rows, N, M2, t, s);
  return cudaGetLastError();
}

}  // namespace gwk

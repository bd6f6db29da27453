// conv.h -- the Bluestein convolution of many FP32 rows (conv.cu).
#pragma once

#include <cuda_runtime.h>

namespace gwk {

// w_M^{j2 k1}, the chirp's spectrum in the order of the middle pass, w_512.
struct ConvTables {
  const float2 *tw, *spec, *tab;
};
// 0 where the length has no kernels (M not a power of two in 2^14 .. 2^18).
size_t conv_table_bytes(int M);
ConvTables conv_tables_at(void *p, int M);
// B: FFT_M of the chirp / M.
cudaError_t launch_conv_tables(const float2 *B, int M, void *p, cudaStream_t s);
// a[row * M + k], k < N, becomes the inverse transform of the rows' transform
// times B at k < N; entries beyond N are scratch.
cudaError_t launch_conv(float2 *a, int rows, int N, int M, const ConvTables &t, cudaStream_t s);

}  // namespace gwk

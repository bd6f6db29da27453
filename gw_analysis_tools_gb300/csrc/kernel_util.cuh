// kernel_util.cuh -- device helpers shared by the kernels' translation units.
#pragma once

#include "kernels.h"

namespace gwk {
using namespace gwt;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Returns true in every thread of the block that finished last.
__device__ __forceinline__ bool arrive_last(unsigned *counter, unsigned expected) {
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned prev = atomicAdd(counter, 1u);
    s_last = (prev == expected - 1);
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Programmatic dependent launch: a kernel launched with the programmatic
// stream-serialisation attribute may start while the one before it on the
// stream still runs; grid_dep_wait() returns once that kernel has completed
// and its memory is visible, and grid_dep_trigger() lets the next kernel start
// launching.  Without the attribute both are no-ops.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }


// The work order of a batch (OrderArgs): the first position of each bucket and,
// past the last, the number of items, by one warp, ...
__device__ __forceinline__ void order_starts(const BatchArgs &a, int *s_bstart) {
  const int tid = threadIdx.x & 31;
  constexpr int kPerLane = (kOrderBuckets + 31) / 32;
  int v[kPerLane], sum = 0;
#pragma unroll
  for (int q = 0; q < kPerLane; q++) {
    const int b = tid * kPerLane + q;
    v[q] = b < kOrderBuckets ? __ldcg(a.bucket_fill + b) : 0;
    sum += v[q];
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (tid >= o) incl += y;
  }
  int run = incl - sum;
#pragma unroll
  for (int q = 0; q < kPerLane; q++) {
    const int b = tid * kPerLane + q;
    if (b < kOrderBuckets) s_bstart[b] = run;
    run += v[q];
  }
  if (tid == 31) s_bstart[kOrderBuckets] = run;
}
// ... and the item at position it (its own index: its partial sums' slot).
__device__ __forceinline__ int order_item(const BatchArgs &a, const int *s_bstart, int it) {
  int iid = it;
  if (a.bucket_fill && it < s_bstart[kOrderBuckets]) {  // the bucket holding position it: the last start <= it
    int lo = 0, hi = kOrderBuckets - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_bstart[mid] <= it) lo = mid;
      else hi = mid - 1;
    }
    iid = __ldcg(a.bucket_items + (size_t)lo * a.nitems + (it - s_bstart[lo]));
  }
  return iid;
}

constexpr int kStatusBounds = 0x100;  // set by an item whose bins fall outside the tables; finalize reports 5

}  // namespace gwk

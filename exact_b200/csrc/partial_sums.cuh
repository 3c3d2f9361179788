// Sum of per-CTA partial rows in a fixed order: the last step of the kernels that reduce over node rows.
//
// 32 adjacent columns per block and kSumSlices threads per column: slice s adds partials s, s + kSumSlices, ... (eight
// loads in flight), the slices are added in order.  With one thread per column walking all partials the step was a chain
// of 1,184 dependent-latency loads on one or two SMs: 98 us behind a 170 MB batch-norm backward, 36 us behind a
// bias gradient; 4 us this way.
#pragma once
#include "common.cuh"

namespace exb {

constexpr int kSumSlices = 16;

// Every thread of a (32, kSumSlices) block calls it; the sum (in the precision of s_part) is returned to the threads of slice 0.
template <typename Sum>
__device__ __forceinline__ Sum sum_partials(const float* __restrict__ column, long long stride, int n, bool valid, Sum (*s_part)[33]) {
  const int sl = threadIdx.y;
  Sum a = 0;
  if (valid) {
    int i = sl;
    for (; i + 7 * kSumSlices < n; i += 8 * kSumSlices) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = column[(long long)(i + u * kSumSlices) * stride];
#pragma unroll
      for (int u = 0; u < 8; u++) a += v[u];
    }
    for (; i < n; i += kSumSlices) a += column[(long long)i * stride];
  }
  __syncthreads();          // s_part may still be read for the previous sum
  s_part[sl][threadIdx.x] = a;
  __syncthreads();
  Sum t = 0;
  if (sl == 0) {
#pragma unroll
    for (int y = 0; y < kSumSlices; y++) t += s_part[y][threadIdx.x];
  }
  return t;
}

}  // namespace exb

// One pass over the gradient of a layer's output for the two things its backward needs besides the GEMMs:
//   colsum[c] = sum_r g[r, c]               the bias gradient (grad_output.sum(0), backward_func.cc:88-90)
//   out[r, c] = g[r, c] * rowscale[r]       D^-1 g, the operand of the transposed mean aggregation
//                                           (A_mean^T g = A^T (D^-1 g), spmm.cc:128-137), zero-padded to Kout columns
// The framework's own route is a broadcast multiply (a non-vectorised element-wise kernel, split in two above
// 2 GB: 1.64 ms at 2,449,029 x 256) and a two-stage column reduction (0.58 ms); this kernel reads g once with
// 16-byte accesses.  Column sums are added in a fixed order (per-CTA partial rows, then those): results are
// run-to-run identical.  A thread owns VEC adjacent columns and walks down the rows.
//
// HALF: the copy is fp16 and unscaled, the operand of the aggregation under autocast: conversion and bias gradient in one
// pass of 30 us at 169,343 x 256, where a conversion and a column sum took 84.
#include <cuda_fp16.h>

#include "exact_b200.h"
#include "common.cuh"
#include "partial_sums.cuh"

namespace exb {

constexpr int kRowOpsThreads = 256;

struct RowOpsParams {
  const float* g;
  const float* rowscale;   // or null (ones)
  void* out;               // or null; fp32 or halves
  float* copy;             // or null; g itself, padded as out is
  float* partial;          // [grid, Kout] or null
  long long n, ldg, ldo;
  int K, Kout, cg_total, cg, ry;
};

template <int VEC, bool HALF>
__global__ void __launch_bounds__(kRowOpsThreads) rows_scale_colsum_kernel(const __grid_constant__ RowOpsParams p) {
  __shared__ float s_red[kRowOpsThreads * VEC];
  const int tx = threadIdx.x % p.cg, ty = threadIdx.x / p.cg;
  const bool active = ty < p.ry;
  for (int cg0 = 0; cg0 < p.cg_total; cg0 += p.cg) {
    const int cgi = cg0 + tx;
    const int c = cgi * VEC;
    const bool col_ok = active && cgi < p.cg_total;
    const bool in_g = c < p.K;            // K is a multiple of VEC, so a group is inside or outside as a whole
    float acc[VEC];
#pragma unroll
    for (int x = 0; x < VEC; x++) acc[x] = 0.f;
    if (col_ok) {
      // four rows per step: four loads in flight per thread (one per step left the kernel waiting on memory:
      // 59 % DRAM throughput at 0.18 issue slots per cycle)
      constexpr int kRowsPerStep = 4;
      const long long rstride = (long long)gridDim.x * p.ry;
      for (long long r0 = (long long)blockIdx.x * p.ry + ty; r0 < p.n; r0 += rstride * kRowsPerStep) {
        float v[kRowsPerStep][VEC], s[kRowsPerStep];
#pragma unroll
        for (int u = 0; u < kRowsPerStep; u++) {
          const long long r = r0 + u * rstride;
#pragma unroll
          for (int x = 0; x < VEC; x++) v[u][x] = 0.f;
          s[u] = 1.f;
          if (r < p.n) {
            if (in_g) Ld<float, VEC>::load(p.g + r * p.ldg + c, v[u]);
            if (p.out != nullptr && p.rowscale != nullptr) s[u] = __ldg(p.rowscale + r);
          }
        }
#pragma unroll
        for (int u = 0; u < kRowsPerStep; u++) {
          const long long r = r0 + u * rstride;
          if (r >= p.n) break;
#pragma unroll
          for (int x = 0; x < VEC; x++) acc[x] = __fadd_rn(acc[x], v[u][x]);
          if (!HALF && p.copy != nullptr) StF32<VEC>::store(p.copy + r * p.ldo + c, v[u]);
          if (p.out != nullptr) {
#pragma unroll
            for (int x = 0; x < VEC; x++) v[u][x] = __fmul_rn(v[u][x], s[u]);
            if (HALF) {
              __half* dst = static_cast<__half*>(p.out) + r * p.ldo + c;
              if constexpr (VEC == 4) {
                const __half2 a = __floats2half2_rn(v[u][0], v[u][1]), b = __floats2half2_rn(v[u][2], v[u][3]);
                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
              } else {
                dst[0] = __float2half_rn(v[u][0]);
              }
            } else {
              StF32<VEC>::store(static_cast<float*>(p.out) + r * p.ldo + c, v[u]);
            }
          }
        }
      }
    }
    if (p.partial != nullptr) {
      float* mine = s_red + threadIdx.x * VEC;
#pragma unroll
      for (int x = 0; x < VEC; x++) mine[x] = acc[x];
      __syncthreads();
      if (ty == 0 && cgi < p.cg_total) {
        float t[VEC];
#pragma unroll
        for (int x = 0; x < VEC; x++) t[x] = 0.f;
        for (int y = 0; y < p.ry; y++) {
#pragma unroll
          for (int x = 0; x < VEC; x++) t[x] = __fadd_rn(t[x], s_red[(y * p.cg + tx) * VEC + x]);
        }
#pragma unroll
        for (int x = 0; x < VEC; x++) p.partial[(long long)blockIdx.x * p.Kout + c + x] = t[x];
      }
      __syncthreads();
    }
  }
}

// Rows padded with zeros to whole 16-byte pieces (and scaled).  Bound by memory; the result is one run of pieces that consecutive
// threads make in order, so no piece of a row is read or written in another pass than its neighbours.  232,965 x 602:
// 196 us; with a thread per column 352, with a thread per pair of columns 300.
template <bool PAIRS>   // rows start on 8-byte boundaries
__global__ void __launch_bounds__(kRowOpsThreads) pad_rows_kernel(const float* __restrict__ g, const float* __restrict__ rowscale,
                                                                  float* __restrict__ out, long long pieces, int K, long long ldg,
                                                                  int per_row) {
  const long long step = (long long)gridDim.x * kRowOpsThreads;
  for (long long i0 = (long long)blockIdx.x * kRowOpsThreads + threadIdx.x; i0 < pieces; i0 += 4 * step) {
    float v[4][4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const long long i = i0 + u * step;
#pragma unroll
      for (int e = 0; e < 4; e++) v[u][e] = 0.f;
      if (i < pieces) {
        const long long r = pieces < (1LL << 32) ? (long long)((uint32_t)i / (uint32_t)per_row) : i / per_row;
        const int c = (int)(i - r * per_row) * 4;
        const float* src = g + r * ldg + c;
        if (PAIRS) {
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            if (c + e + 1 < K) {
              const float2 t = __ldg(reinterpret_cast<const float2*>(src + e));
              v[u][e] = t.x;
              v[u][e + 1] = t.y;
            } else if (c + e < K) {
              v[u][e] = __ldg(src + e);
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (c + e < K) v[u][e] = __ldg(src + e);
        }
        if (rowscale != nullptr) {
          const float s = __ldg(rowscale + r);
#pragma unroll
          for (int e = 0; e < 4; e++) v[u][e] = __fmul_rn(v[u][e], s);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const long long i = i0 + u * step;
      if (i < pieces) __stcs(reinterpret_cast<float4*>(out) + i, make_float4(v[u][0], v[u][1], v[u][2], v[u][3]));
    }
  }
}

__global__ void __launch_bounds__(32 * kSumSlices) rows_colsum_finish_kernel(const float* __restrict__ partial, int n_partial,
                                                                             int K, int Kout, float* __restrict__ colsum) {
  __shared__ float s_part[kSumSlices][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  const float a = sum_partials(partial + c, Kout, n_partial, c < K, s_part);
  if (threadIdx.y == 0 && c < K) colsum[c] = a;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_rows_scale_colsum_workspace_bytes(int64_t Kout) {
  if (Kout <= 0) return 256;
  return 256 + (int64_t)sm_count() * 8 * Kout * 4;
}

static int rows_pass(const float* g, int64_t n, int64_t K, int64_t ldg, const float* rowscale, void* out, float* copy, bool half, int64_t Kout,
                     int64_t ldo, float* colsum, void* workspace, int64_t workspace_bytes, void* stream) {
  EXB_REQUIRE(n >= 0 && K > 0 && ldg >= K, "rows_scale_colsum: bad shape");
  EXB_REQUIRE(K <= (1 << 20), "rows_scale_colsum: too many columns");
  if (out == nullptr) Kout = K;
  EXB_REQUIRE(Kout >= K && (out == nullptr || ldo >= Kout), "rows_scale_colsum: out must hold at least K columns per row");
  EXB_REQUIRE(g != nullptr && (out != nullptr || colsum != nullptr), "rows_scale_colsum: null pointer");
  if (colsum != nullptr) {
    EXB_REQUIRE(workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0 &&
                    workspace_bytes >= exact_rows_scale_colsum_workspace_bytes(Kout),
                "rows_scale_colsum: workspace missing, misaligned or too small");
  }
  cudaStream_t st = (cudaStream_t)stream;
  uintptr_t a = reinterpret_cast<uintptr_t>(g) | (uintptr_t)(ldg * 4);
  if (out != nullptr) a |= (reinterpret_cast<uintptr_t>(out) | (uintptr_t)(ldo * (half ? 2 : 4))) * (half ? 2 : 1);
  if (copy != nullptr) a |= reinterpret_cast<uintptr_t>(copy);
  const bool vec = K % 4 == 0 && Kout % 4 == 0 && a % 16 == 0;
  const int V = vec ? 4 : 1;
  if (!vec && !half && colsum == nullptr && copy == nullptr && Kout % 4 == 0 && ldo == Kout &&
      (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    // rows that only need padding (without column sums nothing ties a thread to its columns)
    const long long pieces = n * (Kout / 4);
    if (pieces == 0) return EXB_OK;
    const bool pairs = (reinterpret_cast<uintptr_t>(g) & 7) == 0 && ldg % 2 == 0;
    auto kernel = pairs ? pad_rows_kernel<true> : pad_rows_kernel<false>;
    const long long want = (pieces + 4 * kRowOpsThreads - 1) / (4 * kRowOpsThreads);
    const int blocks = pairs ? resident_blocks<pad_rows_kernel<true>>(kRowOpsThreads, want)
                             : resident_blocks<pad_rows_kernel<false>>(kRowOpsThreads, want);
    kernel<<<blocks, kRowOpsThreads, 0, st>>>(g, rowscale, static_cast<float*>(out), pieces, (int)K, ldg, (int)(Kout / 4));
    EXB_CUDA_OK(cudaGetLastError());
    return EXB_OK;
  }
  RowOpsParams p{};
  p.g = g; p.rowscale = rowscale; p.out = out; p.copy = copy; p.n = n; p.ldg = ldg; p.ldo = ldo; p.K = (int)K; p.Kout = (int)Kout;
  p.partial = colsum != nullptr ? reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256) : nullptr;
  p.cg_total = (int)((Kout + V - 1) / V);
  const int rounds = (p.cg_total + kRowOpsThreads / V - 1) / (kRowOpsThreads / V);
  p.cg = (p.cg_total + rounds - 1) / rounds;      // equal shares of a row wider than the CTA
  p.ry = kRowOpsThreads / p.cg;
  long long want = (n + p.ry - 1) / p.ry;
  const long long cap = (long long)sm_count() * 8;
  if (want > cap) want = cap;
  const int grid = (int)(want < 1 ? 1 : want);
  if (half) {
    if (vec) rows_scale_colsum_kernel<4, true><<<grid, kRowOpsThreads, 0, st>>>(p);
    else rows_scale_colsum_kernel<1, true><<<grid, kRowOpsThreads, 0, st>>>(p);
  } else {
    if (vec) rows_scale_colsum_kernel<4, false><<<grid, kRowOpsThreads, 0, st>>>(p);
    else rows_scale_colsum_kernel<1, false><<<grid, kRowOpsThreads, 0, st>>>(p);
  }
  EXB_CUDA_OK(cudaGetLastError());
  if (colsum != nullptr) {
    rows_colsum_finish_kernel<<<(unsigned)((K + 31) / 32), dim3(32, kSumSlices), 0, st>>>(p.partial, grid, (int)K, (int)Kout, colsum);
    EXB_CUDA_OK(cudaGetLastError());
  }
  return EXB_OK;
}

int exact_rows_scale_colsum(const float* g, int64_t n, int64_t K, int64_t ldg, const float* rowscale, float* out,
                            int64_t Kout, int64_t ldo, float* colsum, void* workspace, int64_t workspace_bytes,
                            void* stream) {
  return rows_pass(g, n, K, ldg, rowscale, out, nullptr, false, Kout, ldo, colsum, workspace, workspace_bytes, stream);
}

int exact_rows_scale_copy_colsum(const float* g, int64_t n, int64_t K, int64_t ldg, const float* rowscale, float* out, float* copy,
                                 int64_t Kout, int64_t ldo, float* colsum, void* workspace, int64_t workspace_bytes, void* stream) {
  EXB_REQUIRE(out != nullptr && copy != nullptr, "rows_scale_copy_colsum: null output");
  return rows_pass(g, n, K, ldg, rowscale, out, copy, false, Kout, ldo, colsum, workspace, workspace_bytes, stream);
}

int exact_rows_half_colsum(const float* g, int64_t n, int64_t K, int64_t ldg, void* out_f16, int64_t Kout, int64_t ldo, float* colsum,
                           void* workspace, int64_t workspace_bytes, void* stream) {
  EXB_REQUIRE(out_f16 != nullptr, "rows_half_colsum: null output");
  return rows_pass(g, n, K, ldg, nullptr, out_f16, nullptr, true, Kout, ldo, colsum, workspace, workspace_bytes, stream);
}

}  // extern "C"

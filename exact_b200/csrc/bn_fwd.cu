// Batch norm of a training step, forward (native_batch_norm as the reference's qbatch_norm calls it: exact/exact/ops.py:222-229,
// backward_func.cc:95-99):
//     y = (x - mean) * invstd * weight + bias,   invstd = 1 / sqrt(var + eps),
// mean and (biased) variance over the rows, and the running statistics moved by `momentum` (the variance unbiased).
//
// Bound by memory: x is read twice and y written once, 12 N D bytes.  The framework's kernels took 93 us for the statistics and
// 71 us for the transform at 169,343 x 256 (173 MB: 27 us a pass), 38 + 14 and 51 us here.
//
// A thread owns four adjacent columns and walks down the rows, four rows in flight.  It sums deviations from its own first row
// and their squares, so that neither the mean's size nor the number of rows costs the variance digits, turns them into (count,
// mean, sum of squared deviations) and the CTA merges its threads' triples; the finish kernel adds the CTAs' in double and in
// a fixed order: run-to-run identical.
#include "exact_b200.h"
#include "common.cuh"

namespace exb {

constexpr int kBnFwdThreads = 256, kBnFwdRows = 4, kBnSlices = 32;

struct BnFwdParams {
  const float* x;
  const float* weight;   // or null (ones)
  const float* bias;     // or null (zeros)
  float* partial;        // [grid, 3, D]: count, mean, M2
  float* y;
  float* mean;
  float* invstd;
  float* running_mean;   // or null
  float* running_var;
  float momentum, eps;
  long long N;
  int D, cg_total, cg, ry;
};

// (na, ma, qa) <- the union with (nb, mb, qb)
__device__ __forceinline__ void merge_moments(float& na, float& ma, float& qa, float nb, float mb, float qb) {
  if (nb == 0.f) return;
  if (na == 0.f) {
    na = nb; ma = mb; qa = qb;
    return;
  }
  const float n = na + nb, delta = mb - ma, f = nb / n;
  ma = __fmaf_rn(delta, f, ma);
  qa += qb + delta * delta * na * f;
  na = n;
}

__global__ void __launch_bounds__(kBnFwdThreads) bn_fwd_stats_kernel(const __grid_constant__ BnFwdParams p) {
  __shared__ float s_red[3][kBnFwdThreads * 4];
  const int tx = threadIdx.x % p.cg, ty = threadIdx.x / p.cg;
  for (int cg0 = 0; cg0 < p.cg_total; cg0 += p.cg) {
    const int d = (cg0 + tx) * 4;
    const bool ok = ty < p.ry && cg0 + tx < p.cg_total;
    float n = 0.f, mean[4] = {0.f, 0.f, 0.f, 0.f}, m2[4] = {0.f, 0.f, 0.f, 0.f};
    const long long first = (long long)blockIdx.x * p.ry + ty, step = (long long)gridDim.x * p.ry;
    if (ok && first < p.N) {
      float shift[4], s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
      const float4 f = __ldg(reinterpret_cast<const float4*>(p.x + first * p.D + d));
      shift[0] = f.x; shift[1] = f.y; shift[2] = f.z; shift[3] = f.w;
      for (long long r0 = first; r0 < p.N; r0 += step * kBnFwdRows) {
        float4 v[kBnFwdRows];
#pragma unroll
        for (int u = 0; u < kBnFwdRows; u++) {
          const long long r = r0 + u * step;
          v[u] = r < p.N ? __ldg(reinterpret_cast<const float4*>(p.x + r * p.D + d)) : f;   // f: a deviation of zero
          n += r < p.N ? 1.f : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kBnFwdRows; u++) {
          const float a[4] = {v[u].x - shift[0], v[u].y - shift[1], v[u].z - shift[2], v[u].w - shift[3]};
#pragma unroll
          for (int c = 0; c < 4; c++) {
            s1[c] += a[c];
            s2[c] = __fmaf_rn(a[c], a[c], s2[c]);
          }
        }
      }
      const float inv = 1.f / n;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        mean[c] = __fmaf_rn(s1[c], inv, shift[c]);
        m2[c] = fmaxf(__fmaf_rn(-s1[c] * inv, s1[c], s2[c]), 0.f);
        if (isnan(s2[c])) m2[c] = s2[c];     // fmaxf would drop it
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      s_red[0][threadIdx.x * 4 + c] = n;
      s_red[1][threadIdx.x * 4 + c] = mean[c];
      s_red[2][threadIdx.x * 4 + c] = m2[c];
    }
    __syncthreads();
    if (ty == 0 && ok) {
      float* dst = p.partial + (long long)blockIdx.x * 3 * p.D + d;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float na = 0.f, ma = 0.f, qa = 0.f;
        for (int y = 0; y < p.ry; y++) {
          const int at = (y * p.cg + tx) * 4 + c;
          merge_moments(na, ma, qa, s_red[0][at], s_red[1][at], s_red[2][at]);
        }
        dst[c] = na;
        dst[p.D + c] = ma;
        dst[2 * p.D + c] = qa;
      }
    }
    __syncthreads();
  }
}

// Statistics of 32 columns per block, from the CTAs' triples: sums of deviations from the first CTA's mean, in double.  A
// thread takes every 32nd triple, four of them in flight: one at a time took 60 us of load latency for 1,184 triples.
__global__ void __launch_bounds__(32 * kBnSlices) bn_fwd_finish_kernel(const __grid_constant__ BnFwdParams p, int n_partial) {
  __shared__ double s_sum[2][kBnSlices][33];
  const int d = blockIdx.x * 32 + threadIdx.x, sl = threadIdx.y;
  const bool ok = d < p.D;
  const float* __restrict__ q = p.partial + (ok ? d : 0);
  const long long stride = 3LL * p.D;
  const double shift = (double)q[p.D];
  double a = 0.0, b = 0.0;
  for (int i0 = sl; i0 < n_partial; i0 += 4 * kBnSlices) {
    float n[4], m[4], m2[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * kBnSlices < n_partial ? i0 + u * kBnSlices : i0;
      n[u] = q[i * stride];
      m[u] = q[i * stride + p.D];
      m2[u] = q[i * stride + 2 * p.D];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (i0 + u * kBnSlices < n_partial && n[u] > 0.f) {
        const double dev = (double)m[u] - shift;
        a += (double)n[u] * dev;
        b += (double)m2[u] + (double)n[u] * dev * dev;
      }
    }
  }
  s_sum[0][sl][threadIdx.x] = a;
  s_sum[1][sl][threadIdx.x] = b;
  __syncthreads();
  if (sl != 0 || !ok) return;
#pragma unroll
  for (int y = 1; y < kBnSlices; y++) {
    a += s_sum[0][y][threadIdx.x];
    b += s_sum[1][y][threadIdx.x];
  }
  const double dev = a / (double)p.N, mean = shift + dev;
  double m2 = b - a * dev;
  if (m2 < 0.0) m2 = 0.0;
  const double var = m2 / (double)p.N;
  p.mean[d] = (float)mean;
  p.invstd[d] = (float)(1.0 / sqrt(var + (double)p.eps));
  if (p.running_mean) {
    p.running_mean[d] = (1.f - p.momentum) * p.running_mean[d] + p.momentum * (float)mean;
    p.running_var[d] = (1.f - p.momentum) * p.running_var[d] + p.momentum * (float)(m2 / (double)(p.N > 1 ? p.N - 1 : 1));
  }
}

__global__ void __launch_bounds__(kBnFwdThreads) bn_fwd_apply_kernel(const __grid_constant__ BnFwdParams p) {
  const int tx = threadIdx.x % p.cg, ty = threadIdx.x / p.cg;
  for (int cg0 = 0; cg0 < p.cg_total; cg0 += p.cg) {
    const int d = (cg0 + tx) * 4;
    if (ty >= p.ry || cg0 + tx >= p.cg_total) continue;
    float mean[4], k[4], b[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      mean[c] = p.mean[d + c];
      k[c] = p.invstd[d + c] * (p.weight ? p.weight[d + c] : 1.f);
      b[c] = p.bias ? p.bias[d + c] : 0.f;
    }
    const long long step = (long long)gridDim.x * p.ry;
    for (long long r0 = (long long)blockIdx.x * p.ry + ty; r0 < p.N; r0 += step * kBnFwdRows) {
      float4 v[kBnFwdRows];
#pragma unroll
      for (int u = 0; u < kBnFwdRows; u++)
        if (r0 + u * step < p.N) v[u] = __ldg(reinterpret_cast<const float4*>(p.x + (r0 + u * step) * p.D + d));
#pragma unroll
      for (int u = 0; u < kBnFwdRows; u++) {
        const long long r = r0 + u * step;
        if (r >= p.N) break;
        __stcs(reinterpret_cast<float4*>(p.y + r * p.D + d),
               make_float4(__fmaf_rn(v[u].x - mean[0], k[0], b[0]), __fmaf_rn(v[u].y - mean[1], k[1], b[1]),
                           __fmaf_rn(v[u].z - mean[2], k[2], b[2]), __fmaf_rn(v[u].w - mean[3], k[3], b[3])));
      }
    }
  }
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_bn_forward_workspace_bytes(int64_t D) { return D > 0 ? (int64_t)sm_count() * 8 * 3 * D * 4 : 256; }

int exact_bn_forward(const float* x, int64_t N, int64_t D, const float* weight, const float* bias, float* running_mean,
                     float* running_var, float momentum, float eps, void* workspace, int64_t workspace_bytes, float* y,
                     float* save_mean, float* save_invstd, void* stream) {
  EXB_REQUIRE(N > 0 && D > 0, "bn_forward: bad shape");
  if (D % 4 != 0 || D > (1 << 20)) return fail(EXB_ERR_UNSUPPORTED, "bn_forward: D = %lld is not a multiple of 4", (long long)D);
  EXB_REQUIRE(x && y && save_mean && save_invstd && workspace, "bn_forward: null pointer");
  EXB_REQUIRE((running_mean != nullptr) == (running_var != nullptr), "bn_forward: running mean and variance go together");
  EXB_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0, "bn_forward: x and y must be 16-byte aligned");
  EXB_REQUIRE(workspace_bytes >= exact_bn_forward_workspace_bytes(D), "bn_forward: workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  BnFwdParams p{};
  p.x = x; p.weight = weight; p.bias = bias; p.partial = static_cast<float*>(workspace); p.y = y; p.mean = save_mean;
  p.invstd = save_invstd; p.running_mean = running_mean; p.running_var = running_var; p.momentum = momentum; p.eps = eps;
  p.N = N; p.D = (int)D;
  p.cg_total = (int)(D / 4);
  p.cg = p.cg_total < 64 ? p.cg_total : 64;
  p.ry = kBnFwdThreads / p.cg;
  long long want = (N + p.ry - 1) / p.ry;
  const long long cap = (long long)sm_count() * 8;
  const int grid = (int)(want < cap ? want : cap);
  bn_fwd_stats_kernel<<<grid, kBnFwdThreads, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  bn_fwd_finish_kernel<<<(unsigned)((D + 31) / 32), dim3(32, kBnSlices), 0, st>>>(p, grid);
  EXB_CUDA_OK(cudaGetLastError());
  bn_fwd_apply_kernel<<<grid, kBnFwdThreads, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // extern "C"

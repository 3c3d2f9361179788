// Batch norm of a training step, forward (native_batch_norm as the reference's qbatch_norm calls it: exact/exact/ops.py:222-229,
// backward_func.cc:95-99):
//     y = (x - mean) * invstd * weight + bias,   invstd = 1 / sqrt(var + eps),
// mean and (biased) variance over the rows, and the running statistics moved by `momentum` (the variance unbiased).
//
// Bound by memory: x is read twice and y written once, 12 N D bytes.  The framework's kernels took 93 us for the statistics and
// 71 us for the transform at 169,343 x 256 (173 MB: 27 us a pass), 34 + 10 and 51 us here.
//
// A thread owns four adjacent columns and walks down the rows, four rows in flight.  It sums deviations from its own first row
// and their squares, so that neither the mean's size nor the number of rows costs the variance digits, turns them into (count,
// mean, sum of squared deviations) and the CTA merges its threads' triples; the finish kernel adds the CTAs' in double and in
// a fixed order: run-to-run identical.
#include "exact_b200.h"
#include "common.cuh"

namespace exb {

constexpr int kBnFwdThreads = 256, kBnFwdRows = 4, kBnSlices = 32, kBnFinish = 8;

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
  // ReLU + dropout behind it
  uint32_t* mask;
  float p, pinv;
  uint32_t off_lo, off_hi;
  unsigned long long q0;
  PhiloxKey key;
  long long live_warps;   // a multiple of what brings a warp back to the same columns
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
// thread takes every 32nd triple, eight of them in flight: one at a time took 60 us of load latency for 1,184 triples.
__global__ void __launch_bounds__(32 * kBnSlices) bn_fwd_finish_kernel(const __grid_constant__ BnFwdParams p, int n_partial) {
  __shared__ double s_sum[2][kBnSlices][33];
  const int d = blockIdx.x * 32 + threadIdx.x, sl = threadIdx.y;
  const bool ok = d < p.D;
  const float* __restrict__ q = p.partial + (ok ? d : 0);
  const long long stride = 3LL * p.D;
  const double shift = (double)q[p.D];
  double a = 0.0, b = 0.0;
  for (int i0 = sl; i0 < n_partial; i0 += kBnFinish * kBnSlices) {
    float n[kBnFinish], m[kBnFinish], m2[kBnFinish];
#pragma unroll
    for (int u = 0; u < kBnFinish; u++) {
      const int i = i0 + u * kBnSlices < n_partial ? i0 + u * kBnSlices : i0;
      n[u] = q[i * stride];
      m[u] = q[i * stride + p.D];
      m2[u] = q[i * stride + 2 * p.D];
    }
#pragma unroll
    for (int u = 0; u < kBnFinish; u++) {
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

// The transform with the ReLU and dropout that follow it, out = dropout(relu(y)), and their common mask: the arithmetic, the noise
// and the mask's layout of the separate kernels (mask.cu), without y.  A warp takes 256 consecutive elements at a time, the next run
// on its way; the number of warps is a multiple of D / gcd(D, 256), so that a lane meets the same columns in every run and
// keeps their constants.  Bound by memory: 8 N D bytes; 169,343 x 256 in 67 us, the two kernels took 51 and 61.
__global__ void __launch_bounds__(256, 3) bn_act_apply_kernel(const __grid_constant__ BnFwdParams p) {
  const int lane = threadIdx.x & 31;
  const long long n = p.N * p.D, nchunks = (n + 255) >> 8;
  long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= p.live_warps) return;
  float mean[8], k[8], b[8];
  {
    int d = (int)(((c << 8) + 8 * lane) % p.D);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      mean[j] = p.mean[d];
      k[j] = p.invstd[d] * (p.weight ? p.weight[d] : 1.f);
      b[j] = p.bias ? p.bias[d] : 0.f;
      if (++d == p.D) d = 0;
    }
  }
  auto load = [&](long long at, float4 (&f)[2]) {     // whole groups of four: D is a multiple of four
    const long long i = (at << 8) + 8 * lane;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      f[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i + 4 * h < n) f[h] = __ldcs(reinterpret_cast<const float4*>(p.x + i + 4 * h));
    }
  };
  float4 next[2];
  load(c, next);
  for (; c < nchunks; c += p.live_warps) {
    const float v[8] = {next[0].x, next[0].y, next[0].z, next[0].w, next[1].x, next[1].y, next[1].z, next[1].w};
    load(c + p.live_warps, next);
    const long long i = (c << 8) + 8 * lane;
    const unsigned long long q = p.q0 + (unsigned long long)((c << 5) + lane);
    uint32_t w[4];
    philox4x32_10((uint32_t)q, (uint32_t)(q >> 32), p.off_lo, p.off_hi, p.key, w);
    float o[8];
    uint32_t word = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float y = __fmaf_rn(v[j] - mean[j], k[j], b[j]), r = y > 0.f ? y : 0.f;
      const bool keep = dropout_uniform((w[j >> 1] >> (16 * (j & 1))) & 0xffffu) > p.p && i + j < n;
      o[j] = __fmul_rn(__fmul_rn(r, keep ? 1.f : 0.f), p.pinv);
      const uint32_t bits = __ballot_sync(0xffffffffu, keep && r > 0.f);
      if (lane == j) word = bits;
    }
    if (lane < 8) p.mask[(c << 3) + lane] = word;
#pragma unroll
    for (int h = 0; h < 8; h += 4)
      if (i + h < n) __stcs(reinterpret_cast<float4*>(p.y + i + h), make_float4(o[h], o[h + 1], o[h + 2], o[h + 3]));
  }
}

// Statistics and running statistics into p.mean / p.invstd; the grid of the statistics' kernel.
static int bn_statistics(BnFwdParams& p, cudaStream_t st, int* grid) {
  p.cg_total = p.D / 4;
  p.cg = p.cg_total < 64 ? p.cg_total : 64;
  p.ry = kBnFwdThreads / p.cg;
  *grid = resident_blocks<bn_fwd_stats_kernel>(kBnFwdThreads, (p.N + p.ry - 1) / p.ry);
  bn_fwd_stats_kernel<<<*grid, kBnFwdThreads, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  bn_fwd_finish_kernel<<<(unsigned)((p.D + 31) / 32), dim3(32, kBnSlices), 0, st>>>(p, *grid);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
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
  int grid = 0;
  const int rc = bn_statistics(p, st, &grid);
  if (rc) return rc;
  bn_fwd_apply_kernel<<<resident_blocks<bn_fwd_apply_kernel>(kBnFwdThreads, (N + p.ry - 1) / p.ry), kBnFwdThreads, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

int exact_bn_act_forward(const float* x, int64_t N, int64_t D, const float* weight, const float* bias, float* running_mean,
                         float* running_var, float momentum, float eps, float prob, uint64_t seed, uint64_t offset,
                         int64_t index_offset, void* workspace, int64_t workspace_bytes, float* out, uint32_t* mask,
                         float* save_mean, float* save_invstd, void* stream) {
  EXB_REQUIRE(N > 0 && D > 0, "bn_act_forward: bad shape");
  EXB_REQUIRE(index_offset >= 0 && index_offset % 8 == 0, "bn_act_forward: index_offset must be a non-negative multiple of 8");
  EXB_REQUIRE(prob >= 0.f && prob <= 1.f, "bn_act_forward: p must be in [0, 1] (got %f)", (double)prob);
  long long period = D;                       // D / gcd(D, 256) runs of 256 elements later a lane is at the same columns
  for (int i = 0; i < 8 && period % 2 == 0; i++) period /= 2;
  const long long nchunks = (N * D + 255) / 256;
  long long warps = 16LL * resident_blocks<bn_act_apply_kernel>(256, 1LL << 40);   // two rounds of blocks: 69 us with one, 67, 69 with four
  if (warps > (nchunks + period) / period * period) warps = (nchunks + period) / period * period;
  if (D % 4 != 0 || D > (1 << 20) || period > warps)
    return fail(EXB_ERR_UNSUPPORTED, "bn_act_forward: no kernel for D = %lld", (long long)D);
  EXB_REQUIRE(x && out && mask && save_mean && save_invstd && workspace, "bn_act_forward: null pointer");
  EXB_REQUIRE((running_mean != nullptr) == (running_var != nullptr), "bn_act_forward: running mean and variance go together");
  EXB_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(mask)) & 15) == 0,
              "bn_act_forward: x, out and mask must be 16-byte aligned");
  EXB_REQUIRE(workspace_bytes >= exact_bn_forward_workspace_bytes(D), "bn_act_forward: workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  BnFwdParams p{};
  p.x = x; p.weight = weight; p.bias = bias; p.partial = static_cast<float*>(workspace); p.y = out; p.mean = save_mean;
  p.invstd = save_invstd; p.running_mean = running_mean; p.running_var = running_var; p.momentum = momentum; p.eps = eps;
  p.N = N; p.D = (int)D; p.mask = mask; p.p = prob; p.pinv = dropout_scale(prob).pinv;
  p.off_lo = (uint32_t)offset; p.off_hi = (uint32_t)(offset >> 32); p.q0 = (unsigned long long)index_offset >> 3;
  p.key = make_philox_key(seed);
  int grid = 0;
  const int rc = bn_statistics(p, st, &grid);
  if (rc) return rc;
  p.live_warps = warps / period * period;
  bn_act_apply_kernel<<<(unsigned)((p.live_warps + 7) / 8), 256, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // extern "C"

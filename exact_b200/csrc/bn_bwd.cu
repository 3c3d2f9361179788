// Batch-norm backward straight from the packed input.
//
// The reference's qbatch_norm.backward (exact/exact/ops.py:235-253) dequantises the saved input into a
// full [N, D] fp32 tensor (dequantize_activation, ops.py:86-98 -> quantization_cuda_kernel.cu:158-185) and
// hands it to native_batch_norm_backward, which reads it twice (the column sums, then the element-wise
// pass).  Here both passes read the packed bytes and the row statistics instead and dequantise in
// registers (code / scale + min, IEEE, the arithmetic of quantization_cuda_kernel.cu:182): the [N, D]
// reconstruction never exists, and the backward moves 12 N D bytes instead of 24 N D.
//
//   pass 1  bn_bwd_kernel           per column d: sum_n g[n, d] and sum_n g[n, d] (x[n, d] - mean[d]); every CTA
//                                   writes its partial sums, bn_bwd_finish_kernel adds them in a fixed order (no float
//                                   atomics: results are run-to-run identical) and forms
//                                   grad_bias = sum g, grad_weight = invstd * sum g (x - mean);
//   pass 2  bn_bwd_kernel           training: grad_in = (g - sum_g / N - (x - mean) * invstd^2 * sum_gx / N) * invstd * w
//                                   eval:     grad_in = g * invstd * w
//
// A thread owns four adjacent columns (one 32-bit word of the packed stream = those columns of 8 / bits
// consecutive rows) and walks down the rows, so its per-column constants stay in registers and every access
// is a 16-byte piece of a row.
#include "exact_b200.h"
#include "common.cuh"
#include "partial_sums.cuh"

namespace exb {

constexpr int kBnThreads = 256;

struct BnBwdParams {
  const float* g;
  const uint8_t* packed;
  const uint16_t* scale_bf16;
  const uint16_t* min_bf16;
  const float* weight;   // or null (ones)
  const float* mean;
  const float* invstd;
  float* partial;        // [grid, 2, D]
  float* sums;           // [2, D]: sum g, sum g (x - mean)
  float* grad_in;
  float* grad_weight;    // or null
  float* grad_bias;      // or null
  long long N;
  int D, cg_total, cg, ry, training;
  long long groups;      // ceil(N / (8 / bits))
  const uint32_t* mask;  // of the ReLU + dropout behind the batch norm (mask.cu's layout); g is the gradient of their output
  float p1m, p1m_inv_exact;
};

// code / s + m, IEEE: by the correctly rounded reciprocal when s is an ordinary number (equal to the quotient
// for every code 0..255 and 2^-100 <= |s| <= 2^100), by the division otherwise (inf of a constant row, NaN,
// denormals).
__device__ __forceinline__ float dequant_one(uint32_t code, float s, float rcp, float m, bool tame) {
  const float c = (float)code;
  if (tame) {
    const float q0 = __fmul_rn(c, rcp);
    const float q = __fmaf_rn(__fmaf_rn(-q0, s, c), rcp, q0);
    return __fadd_rn(q, m);
  }
  return __fadd_rn(__fdiv_rn(c, s), m);
}

template <int BITS, bool APPLY, bool MASKED>
__global__ void __launch_bounds__(kBnThreads) bn_bwd_kernel(const __grid_constant__ BnBwdParams p) {
  constexpr int WPT = 8 / BITS;
  constexpr uint32_t MASK = (1u << BITS) - 1u;
  __shared__ float s_red[APPLY ? 1 : kBnThreads * 8];
  const int tx = threadIdx.x % p.cg, ty = threadIdx.x / p.cg;
  const bool active = ty < p.ry;
  for (int cg0 = 0; cg0 < p.cg_total; cg0 += p.cg) {
    const int cgi = cg0 + tx;
    const bool col_ok = active && cgi < p.cg_total;
    const int d = cgi * 4;
    float mean[4] = {0.f, 0.f, 0.f, 0.f}, k2[4] = {0.f, 0.f, 0.f, 0.f}, k1[4] = {0.f, 0.f, 0.f, 0.f},
          gs[4] = {0.f, 0.f, 0.f, 0.f};
    if (col_ok) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        mean[c] = p.mean[d + c];
        if (APPLY) {
          const float is = p.invstd[d + c];
          gs[c] = __fmul_rn(is, p.weight ? p.weight[d + c] : 1.f);
          if (p.training) {
            const float inv_n = 1.f / (float)p.N;
            k1[c] = __fmul_rn(p.sums[d + c], inv_n);
            k2[c] = __fmul_rn(__fmul_rn(p.sums[p.D + d + c], inv_n), __fmul_rn(is, is));
          }
        }
      }
    }
    float acc_g[4] = {0.f, 0.f, 0.f, 0.f}, acc_gx[4] = {0.f, 0.f, 0.f, 0.f};
    if (col_ok) {
      for (long long grp = (long long)blockIdx.x * p.ry + ty; grp < p.groups; grp += (long long)gridDim.x * p.ry) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(p.packed + grp * p.D + d));
        const long long n0 = grp * WPT;
        float4 gv[WPT];
        uint4 mv[MASKED ? WPT : 1];
        float s[WPT], m[WPT];
#pragma unroll
        for (int i = 0; i < WPT; i++) {
          const long long n = n0 + i;
          if (n < p.N) {
            gv[i] = __ldcs(reinterpret_cast<const float4*>(p.g + n * p.D + d));
            // element e: bit (e >> 3) & 31 of word 8 (e >> 8) + (e & 7)
            if (MASKED) mv[MASKED ? i : 0] = __ldg(reinterpret_cast<const uint4*>(p.mask) + ((n * p.D + d) >> 8) * 2 + ((d + n * p.D) >> 2 & 1));
            s[i] = bf16_bits_to_f32(__ldg(p.scale_bf16 + n));
            m[i] = bf16_bits_to_f32(__ldg(p.min_bf16 + n));
          } else {
            gv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            s[i] = 1.f;
            m[i] = 0.f;
          }
        }
#pragma unroll
        for (int i = 0; i < WPT; i++) {
          const long long n = n0 + i;
          if (n >= p.N) break;
          const uint32_t sexp = (__float_as_uint(s[i]) >> 23) & 0xffu;
          const bool tame = sexp >= 27u && sexp <= 227u;
          const float rcp = __frcp_rn(s[i]);
          float gg[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w};
          if (MASKED) {
            const uint32_t bit = 1u << ((unsigned)(n * p.D + d) >> 3 & 31u);
            const uint4 mk = mv[MASKED ? i : 0];
            const uint32_t mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
            for (int c = 0; c < 4; c++) gg[c] = (mw[c] & bit) ? dropout_grad(gg[c], p.p1m, p.p1m_inv_exact) : 0.f;
          }
          float o[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const uint32_t code = ((w >> (8 * c)) >> (i * BITS)) & MASK;
            const float xc = __fsub_rn(dequant_one(code, s[i], rcp, m[i], tame), mean[c]);
            if (APPLY) {
              o[c] = p.training ? __fmul_rn(__fsub_rn(__fsub_rn(gg[c], k1[c]), __fmul_rn(xc, k2[c])), gs[c])
                                : __fmul_rn(gg[c], gs[c]);
            } else {
              acc_g[c] = __fadd_rn(acc_g[c], gg[c]);
              acc_gx[c] = __fmaf_rn(gg[c], xc, acc_gx[c]);
            }
          }
          if (APPLY) __stcs(reinterpret_cast<float4*>(p.grad_in + n * p.D + d), make_float4(o[0], o[1], o[2], o[3]));
        }
      }
    }
    if (!APPLY) {
      // add the row lanes of each column group in lane order, one partial row per CTA
      float* mine = s_red + threadIdx.x * 8;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        mine[c] = acc_g[c];
        mine[4 + c] = acc_gx[c];
      }
      __syncthreads();
      if (ty == 0 && cgi < p.cg_total) {
        float tg[4] = {0.f, 0.f, 0.f, 0.f}, tgx[4] = {0.f, 0.f, 0.f, 0.f};
        for (int y = 0; y < p.ry; y++) {
          const float* o = s_red + (y * p.cg + tx) * 8;
#pragma unroll
          for (int c = 0; c < 4; c++) {
            tg[c] = __fadd_rn(tg[c], o[c]);
            tgx[c] = __fadd_rn(tgx[c], o[4 + c]);
          }
        }
        float* dst = p.partial + (long long)blockIdx.x * 2 * p.D;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          dst[d + c] = tg[c];
          dst[p.D + d + c] = tgx[c];
        }
      }
      __syncthreads();
    }
  }
}

// The same for widths that are a multiple of eight, the layers' own: a thread owns eight adjacent columns, so that a row's
// reciprocal, statistics and mask words (one run of eight elements has one bit position) serve twice the elements, and the
// arithmetic is paired.  Every element goes through the operations of bn_bwd_kernel.  Bound by memory: 4 N D bytes in, and out for
// the second pass; 169,343 x 256, INT2, behind ReLU + dropout: 47 and 63 us; the kernel above takes 70
// and 95 (48 and 70 without the mask, and 58 for the mask by itself).
template <int BITS, bool APPLY, bool MASKED>
__global__ void __launch_bounds__(kBnThreads, 2) bn_bwd8_kernel(const __grid_constant__ BnBwdParams p) {
  constexpr int WPT = 8 / BITS, R = WPT < 4 ? WPT : 4;   // rows of a byte; rows a thread takes at a time
  constexpr uint32_t MASK = 0x01010101u * ((1u << BITS) - 1u);
  __shared__ float s_red[APPLY ? 1 : kBnThreads * 16];
  const int tx = threadIdx.x % p.cg, ty = threadIdx.x / p.cg;
  const bool active = ty < p.ry;
  for (int cg0 = 0; cg0 < p.cg_total; cg0 += p.cg) {
    const int cgi = cg0 + tx;
    const bool col_ok = active && cgi < p.cg_total;
    const int d = cgi * 8;
    f32x2 mean[4], k1[4], k2[4], gs[4], acc_g[4], acc_gx[4];
#pragma unroll
    for (int c = 0; c < 4; c++) mean[c] = k1[c] = k2[c] = gs[c] = acc_g[c] = acc_gx[c] = f2_pack(0.f, 0.f);
    if (col_ok) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float a[2], b[2], e[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int at = d + 2 * c + h;
          const float is = p.invstd[at], inv_n = 1.f / (float)p.N;
          a[h] = __fmul_rn(is, p.weight ? p.weight[at] : 1.f);
          b[h] = APPLY && p.training ? __fmul_rn(p.sums[at], inv_n) : 0.f;
          e[h] = APPLY && p.training ? __fmul_rn(__fmul_rn(p.sums[p.D + at], inv_n), __fmul_rn(is, is)) : 0.f;
        }
        mean[c] = f2_pack(p.mean[d + 2 * c], p.mean[d + 2 * c + 1]);
        gs[c] = f2_pack(a[0], a[1]);
        k1[c] = f2_pack(b[0], b[1]);
        k2[c] = f2_pack(e[0], e[1]);
      }
      for (long long n0 = ((long long)blockIdx.x * p.ry + ty) * R; n0 < p.N; n0 += (long long)gridDim.x * p.ry * R) {
        uint2 w = __ldg(reinterpret_cast<const uint2*>(p.packed + n0 / WPT * p.D + d));
        if (R < WPT && (n0 & R)) {       // the byte's upper rows
          w.x >>= R * BITS;
          w.y >>= R * BITS;
        }
        const int rows = p.N - n0 < R ? (int)(p.N - n0) : R;
        float4 gv[R][2];
        uint4 mv[MASKED ? R : 1][2];
        float s[R], m[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
          const long long e = (n0 + (i < rows ? i : 0)) * p.D + d;        // rows past the end: the first again, not used
          gv[i][0] = __ldcs(reinterpret_cast<const float4*>(p.g + e));
          gv[i][1] = __ldcs(reinterpret_cast<const float4*>(p.g + e) + 1);
          if (MASKED) {   // element e: bit (e >> 3) & 31 of word 8 (e >> 8) + (e & 7)
            mv[MASKED ? i : 0][0] = __ldg(reinterpret_cast<const uint4*>(p.mask) + (e >> 8) * 2);
            mv[MASKED ? i : 0][1] = __ldg(reinterpret_cast<const uint4*>(p.mask) + (e >> 8) * 2 + 1);
          }
          s[i] = bf16_bits_to_f32(__ldg(p.scale_bf16 + n0 + (i < rows ? i : 0)));
          m[i] = bf16_bits_to_f32(__ldg(p.min_bf16 + n0 + (i < rows ? i : 0)));
        }
#pragma unroll
        for (int i = 0; i < R; i++) {
          if (i >= rows) break;
          const uint32_t sexp = (__float_as_uint(s[i]) >> 23) & 0xffu;
          const bool tame = sexp >= 27u && sexp <= 227u;
          const float rcp = __frcp_rn(s[i]);
          const float gg[8] = {gv[i][0].x, gv[i][0].y, gv[i][0].z, gv[i][0].w, gv[i][1].x, gv[i][1].y, gv[i][1].z, gv[i][1].w};
          f32x2 g2[4], o[4];
          if (MASKED) {
            const uint32_t bit = 1u << ((unsigned)((n0 + i) * p.D + d) >> 3 & 31u);
            const uint4 ma = mv[MASKED ? i : 0][0], mb = mv[MASKED ? i : 0][1];
            const uint32_t mw[8] = {ma.x, ma.y, ma.z, ma.w, mb.x, mb.y, mb.z, mb.w};
            float k[8];
#pragma unroll
            for (int c = 0; c < 8; c++) k[c] = (mw[c] & bit) ? dropout_grad(gg[c], p.p1m, p.p1m_inv_exact) : 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++) g2[c] = f2_pack(k[2 * c], k[2 * c + 1]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; c++) g2[c] = f2_pack(gg[2 * c], gg[2 * c + 1]);
          }
          const uint32_t code[2] = {(w.x >> (i * BITS)) & MASK, (w.y >> (i * BITS)) & MASK};
#pragma unroll
          for (int c = 0; c < 4; c++) {
            // 2^23 + code by one byte permute, exact
            const uint32_t word = code[c >> 1];
            const f32x2 c2 = f2_add(f2_pack(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + (c & 1) * 2)),
                                            __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7541u + (c & 1) * 2))),
                                    f2_pack(-8388608.f, -8388608.f));
            f32x2 x;
            if (tame) {
              const f32x2 r2 = f2_pack(rcp, rcp), q0 = f2_mul(c2, r2);
              const f32x2 rem = f2_fma(q0, f2_pack(-s[i], -s[i]), c2);
              x = f2_add(f2_fma(rem, r2, q0), f2_pack(m[i], m[i]));
            } else {
              float a, b;
              f2_unpack(c2, a, b);
              x = f2_pack(__fadd_rn(__fdiv_rn(a, s[i]), m[i]), __fadd_rn(__fdiv_rn(b, s[i]), m[i]));
            }
            const f32x2 xc = f2_sub(x, mean[c]);
            if (APPLY) {
              o[c] = p.training ? f2_mul(f2_sub(f2_sub(g2[c], k1[c]), f2_mul(xc, k2[c])), gs[c]) : f2_mul(g2[c], gs[c]);
            } else {
              acc_g[c] = f2_add(acc_g[c], g2[c]);
              acc_gx[c] = f2_fma(g2[c], xc, acc_gx[c]);
            }
          }
          if (APPLY) {
            float4* dst = reinterpret_cast<float4*>(p.grad_in + (n0 + i) * p.D + d);
            float a[8];
#pragma unroll
            for (int c = 0; c < 4; c++) f2_unpack(o[c], a[2 * c], a[2 * c + 1]);
            __stcs(dst, make_float4(a[0], a[1], a[2], a[3]));
            __stcs(dst + 1, make_float4(a[4], a[5], a[6], a[7]));
          }
        }
      }
    }
    if (!APPLY) {
      // add the row lanes of each column group in lane order, one partial row per CTA
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float a, b, e, f;
        f2_unpack(acc_g[c], a, b);
        f2_unpack(acc_gx[c], e, f);
        s_red[(4 * c + 0) * kBnThreads + threadIdx.x] = a;
        s_red[(4 * c + 1) * kBnThreads + threadIdx.x] = b;
        s_red[(4 * c + 2) * kBnThreads + threadIdx.x] = e;
        s_red[(4 * c + 3) * kBnThreads + threadIdx.x] = f;
      }
      __syncthreads();
      // thread (tx, v) of the CTA adds value v of column group tx: 16 values, four columns pairs of (g, g x)
      float* dst = p.partial + (long long)blockIdx.x * 2 * p.D;
      for (int at = threadIdx.x; at < 16 * p.cg; at += kBnThreads) {
        const int v = at / p.cg, t = at - v * p.cg;
        if (cg0 + t >= p.cg_total) continue;
        float a = 0.f;
        for (int y = 0; y < p.ry; y++) a = __fadd_rn(a, s_red[v * kBnThreads + y * p.cg + t]);
        dst[(v & 2 ? p.D : 0) + (cg0 + t) * 8 + (v >> 2) * 2 + (v & 1)] = a;
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(32 * kSumSlices) bn_bwd_finish_kernel(
    const float* __restrict__ partial, int n_partial, int D, const float* __restrict__ invstd, float* __restrict__ sums,
    float* __restrict__ grad_weight, float* __restrict__ grad_bias) {
  __shared__ float s_part[kSumSlices][33];
  const int d = blockIdx.x * 32 + threadIdx.x;
  const float a = sum_partials(partial + d, 2LL * D, n_partial, d < D, s_part);
  const float b = sum_partials(partial + D + d, 2LL * D, n_partial, d < D, s_part);
  if (threadIdx.y != 0 || d >= D) return;
  sums[d] = a;
  sums[D + d] = b;
  if (grad_bias) grad_bias[d] = a;
  if (grad_weight) grad_weight[d] = __fmul_rn(b, invstd[d]);
}

template <int BITS, bool APPLY, bool MASKED>
static int launch_bn_bwd(BnBwdParams p, cudaStream_t st) {
  const bool wide = p.D % 8 == 0 && (reinterpret_cast<uintptr_t>(p.packed) & 7) == 0;
  auto kernel = wide ? bn_bwd8_kernel<BITS, APPLY, MASKED> : bn_bwd_kernel<BITS, APPLY, MASKED>;
  p.cg_total = p.D / (wide ? 8 : 4);
  p.cg = p.cg_total < 64 ? p.cg_total : 64;
  p.ry = kBnThreads / p.cg;
  const long long units = wide && BITS == 1 ? 2 * p.groups : p.groups;
  // one grid with a mask and without: the order of the sums, and with it their last bits, does not depend on it
  const long long want = (units + p.ry - 1) / p.ry;
  const int grid = wide ? resident_blocks<bn_bwd8_kernel<BITS, APPLY, true>>(kBnThreads, want)
                        : resident_blocks<bn_bwd_kernel<BITS, APPLY, true>>(kBnThreads, want);
  kernel<<<grid, kBnThreads, 0, st>>>(p);
  return grid;
}
template <bool APPLY>
static int launch_bn_bwd_bits(const BnBwdParams& p, int bits, cudaStream_t st) {
  switch (bits) {
    case 1: return p.mask ? launch_bn_bwd<1, APPLY, true>(p, st) : launch_bn_bwd<1, APPLY, false>(p, st);
    case 2: return p.mask ? launch_bn_bwd<2, APPLY, true>(p, st) : launch_bn_bwd<2, APPLY, false>(p, st);
    case 4: return p.mask ? launch_bn_bwd<4, APPLY, true>(p, st) : launch_bn_bwd<4, APPLY, false>(p, st);
  }
  return p.mask ? launch_bn_bwd<8, APPLY, true>(p, st) : launch_bn_bwd<8, APPLY, false>(p, st);
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_bn_backward_workspace_bytes(int64_t D) {
  if (D <= 0) return 256;
  return 256 + ((int64_t)sm_count() * 8 + 1) * 2 * D * 4;
}

// mask: null, or the ReLU + dropout between the batch norm and grad_out
static int bn_backward(const float* grad_out, const uint32_t* mask, float prob, int64_t N, int64_t D, const uint8_t* packed, int bits,
                       const uint16_t* scale_bf16, const uint16_t* min_bf16, const float* weight, const float* mean,
                       const float* invstd, int training, void* workspace, int64_t workspace_bytes, float* grad_input,
                       float* grad_weight, float* grad_bias, void* stream) {
  EXB_REQUIRE(bits == 1 || bits == 2 || bits == 4 || bits == 8, "bits must be 1, 2, 4 or 8 (got %d)", bits);
  EXB_REQUIRE(N >= 0 && D > 0, "bn_backward_from_packed: bad shape");
  if (D % 4 != 0 || D > (1 << 20))
    return fail(EXB_ERR_UNSUPPORTED, "bn_backward_from_packed: D = %lld is not a multiple of 4", (long long)D);
  EXB_REQUIRE(grad_out && packed && scale_bf16 && min_bf16 && mean && invstd && workspace,
              "bn_backward_from_packed: null pointer");
  EXB_REQUIRE(workspace_bytes >= exact_bn_backward_workspace_bytes(D), "bn_backward_from_packed: workspace too small");
  EXB_REQUIRE(((reinterpret_cast<uintptr_t>(grad_out) | reinterpret_cast<uintptr_t>(grad_input)) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(packed) & 3) == 0 && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0,
              "bn_backward_from_packed: grad_out / grad_input must be 16-byte, packed 4-byte, workspace 256-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  BnBwdParams p{};
  p.g = grad_out; p.packed = packed; p.scale_bf16 = scale_bf16; p.min_bf16 = min_bf16; p.weight = weight;
  p.mean = mean; p.invstd = invstd; p.grad_in = grad_input; p.grad_weight = grad_weight; p.grad_bias = grad_bias;
  p.N = N; p.D = (int)D; p.training = training != 0;
  const int wpt = 8 / bits;
  p.groups = (N + wpt - 1) / wpt;
  p.sums = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  p.partial = p.sums + 2 * D;
  p.mask = mask;
  const DropoutScale drop = dropout_scale(prob);
  p.p1m = drop.p1m;
  p.p1m_inv_exact = drop.p1m_inv_exact;
  if (grad_weight || grad_bias || (grad_input && p.training)) {
    const int grid = launch_bn_bwd_bits<false>(p, bits, st);
    EXB_CUDA_OK(cudaGetLastError());
    bn_bwd_finish_kernel<<<(unsigned)((D + 31) / 32), dim3(32, kSumSlices), 0, st>>>(p.partial, grid, (int)D, invstd, p.sums, grad_weight,
                                                                     grad_bias);
    EXB_CUDA_OK(cudaGetLastError());
  }
  if (grad_input && N > 0) {
    launch_bn_bwd_bits<true>(p, bits, st);
    EXB_CUDA_OK(cudaGetLastError());
  }
  return EXB_OK;
}


int exact_bn_backward_from_packed(const float* grad_out, int64_t N, int64_t D, const uint8_t* packed, int bits,
                                  const uint16_t* scale_bf16, const uint16_t* min_bf16, const float* weight,
                                  const float* mean, const float* invstd, int training, void* workspace,
                                  int64_t workspace_bytes, float* grad_input, float* grad_weight, float* grad_bias,
                                  void* stream) {
  return bn_backward(grad_out, nullptr, 0.f, N, D, packed, bits, scale_bf16, min_bf16, weight, mean, invstd, training, workspace,
                     workspace_bytes, grad_input, grad_weight, grad_bias, stream);
}

int exact_bn_act_backward_from_packed(const float* grad_out, const uint32_t* mask, float prob, int64_t N, int64_t D,
                                      const uint8_t* packed, int bits, const uint16_t* scale_bf16, const uint16_t* min_bf16,
                                      const float* weight, const float* mean, const float* invstd, void* workspace,
                                      int64_t workspace_bytes, float* grad_input, float* grad_weight, float* grad_bias,
                                      void* stream) {
  EXB_REQUIRE(mask != nullptr && (reinterpret_cast<uintptr_t>(mask) & 15) == 0, "bn_act_backward_from_packed: null or misaligned mask");
  EXB_REQUIRE(prob >= 0.f && prob <= 1.f, "bn_act_backward_from_packed: p must be in [0, 1] (got %f)", (double)prob);
  return bn_backward(grad_out, mask, prob, N, D, packed, bits, scale_bf16, min_bf16, weight, mean, invstd, 1, workspace,
                     workspace_bytes, grad_input, grad_weight, grad_bias, stream);
}

}  // extern "C"

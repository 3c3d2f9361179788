// CSR SpMM on fp16 operands with the arithmetic of the reference's half instantiation.
//
// The reference dispatches spmm_kernel on half as well (exact/exact/cpp_extension/spmm_cuda.cu:142, AMP runs:
// exact/exact/ops.py:260, 313 cast the operands to fp16).  With scalar_t = c10::Half every step of the row sum is
// rounded to half (spmm_cuda.cu:83-92, reducer.cuh:53-60, 72-77):
//     term   = half(value[e] * mat[col[e], c])            (with edge values; the bare operand otherwise)
//     result = half(result + term)                        in edge order, starting from 0
//     mean:    out = half(result / half(max(count, 1)))   (the count itself is rounded to half first)
// each Half (op) Half being an fp32 operation on the widened values.  fp32 keeps 24 bits, more than 2 * 11 + 2, so
// rounding the fp32 sum or product of two halves to half gives the correctly rounded half sum or product: the
// paired half instructions (never contracted to an FMA) compute the same bits.
//
// Rounding after every edge makes the order of the edges part of the result, so a row's sum is a chain of one add per
// edge that nothing can cut.  What bounds the kernel is the latency between an edge's index and its add; the two
// kinds of rows are built around keeping gathers in flight ahead of the chain:
//   rows       a group of LPE lanes (the operand row as 16-byte pieces) walks a row, eight gathers per lane at a time;
//              32 warps per SM, which hides more than longer batches or rows prefetched ahead did (24 warps: 141 against
//              138 us, 16 warps with batches of 16: 172 us at 1.78 M edges x 256 columns in rows of up to 256).
//   long rows  (power-law hubs: 10^3 .. 10^5 edges) two warps per 64 columns: one gathers by cp.async into a ring of 256
//              edges, the other adds, so that the chain waits for its own adds and not for memory.  Longest rows
//              first, in a kernel of their own that the rows' kernel does not wait for (programmatic launch).
// 169,343 nodes / 2.54 M edges (R-MAT, longest row 10,679), 256 columns with edge values: 171 us, where one warp walking
// every row took 1,850 us; 40 columns 107 us against 1,750 us (bound by the longest row's chain, 9 ns an edge).
#include <cuda_fp16.h>

#include "exact_b200.h"
#include "common.cuh"

namespace exb {

struct SpmmF16Params {
  const void* rowptr;
  const void* col;
  const __half* val;
  const __half* mat;
  void* out;                  // halves, or fp32 with a bias
  const float* bias;          // [K] added to every row in fp32, or null
  long long M, K, ldm;
  int mean;
  long long long_threshold;   // rows with more edges are left to the hub warps (0: none)
  const int* row_order;       // the order in which the rows are taken, or null
  const int* long_row;        // the rows above the threshold, longest first
  long long n_long;
  long long hub_units;        // n_long x 64-column blocks
};

constexpr int kF16Warps = 8;
constexpr int kHubPairs = 2;          // pairs of warps of a block that take long rows
constexpr int kHubChunks = 4;         // ring of 4 x 64 edges x 128 bytes per pair; 2 pairs x 2 x 4 barriers are all there are
constexpr int kHubRing = kHubChunks * 64 * 128;
constexpr int kF16Smem = kHubPairs * (kHubRing + kHubChunks * 64 * 4);

__device__ __forceinline__ float rh(float f) { return __half2float(__float2half_rn(f)); }

// Pairs of halves in 32-bit registers.  The explicit .rn keeps the two roundings apart (no contraction to an FMA).
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_both(uint32_t low) { return __byte_perm(low, low, 0x1010); }
__device__ __forceinline__ uint32_t h2_mean(uint32_t a, float dv) {
  const float lo = __half2float(__ushort_as_half((unsigned short)(a & 0xffff)));
  const float hi = __half2float(__ushort_as_half((unsigned short)(a >> 16)));
  return (uint32_t)__half_as_ushort(__float2half_rn(__fdiv_rn(lo, dv))) |
         (uint32_t)__half_as_ushort(__float2half_rn(__fdiv_rn(hi, dv))) << 16;
}

template <int VEC>
__device__ __forceinline__ void load_piece(const __half* p, uint32_t (&m)[VEC == 8 ? 4 : 1]) {
  if constexpr (VEC == 8) {
    const uint4 t = __ldg(reinterpret_cast<const uint4*>(p));
    m[0] = t.x; m[1] = t.y; m[2] = t.z; m[3] = t.w;
  } else {
    m[0] = __ldg(reinterpret_cast<const unsigned short*>(p));
  }
}

// acc += terms of edges [t, t + B) of the LPE edges whose indices and values the group holds in `idx` and `val`.
template <int B, bool HAS_VAL, int VEC, int LPE>
__device__ __forceinline__ void f16_edges(const __half* __restrict__ mat0, unsigned long long ldm, uint32_t idx, uint32_t val,
                                          int t, int left, bool cvalid, uint32_t (&acc)[VEC == 8 ? 4 : 1]) {
  constexpr int NH = VEC == 8 ? 4 : 1;
  uint32_t m[B][NH];
#pragma unroll
  for (int u = 0; u < B; u++) {
    const uint32_t j = __shfl_sync(0xffffffffu, idx, t + u, LPE);
#pragma unroll
    for (int x = 0; x < NH; x++) m[u][x] = 0;
    if (t + u < left && cvalid) load_piece<VEC>(mat0 + (unsigned long long)j * ldm, m[u]);
  }
#pragma unroll
  for (int u = 0; u < B; u++) {
    uint32_t w = 0;
    if (HAS_VAL) w = h2_both(__shfl_sync(0xffffffffu, val, t + u, LPE));
    if (t + u < left) {
#pragma unroll
      for (int x = 0; x < NH; x++) acc[x] = h2_add(acc[x], HAS_VAL ? h2_mul(w, m[u][x]) : m[u][x]);
    }
  }
}

template <typename IdxT, bool HAS_VAL, int VEC, int LPE>
__global__ void __launch_bounds__(kF16Warps * 32, 4) spmm_f16_rows_kernel(const __grid_constant__ SpmmF16Params p) {
  constexpr int NH = VEC == 8 ? 4 : 1;
  constexpr int kRows = 32 / LPE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hl = lane % LPE;
  const IdxT* __restrict__ rowptr = static_cast<const IdxT*>(p.rowptr);
  const IdxT* __restrict__ col = static_cast<const IdxT*>(p.col);
  const long long c = (long long)blockIdx.y * (LPE * VEC) + (long long)hl * VEC;
  const bool cvalid = c < p.K;
  const __half* __restrict__ mat0 = p.mat + (cvalid ? c : 0);
  const long long unit = ((long long)blockIdx.x * kF16Warps + warp) * kRows + lane / LPE;

  long long row = -1, b = 0;
  int len = 0;
  if (unit < p.M) {
    row = p.row_order ? (long long)p.row_order[unit] : unit;
    b = (long long)rowptr[row];
    const long long n = (long long)rowptr[row + 1] - b;
    if (p.long_threshold > 0 && n > p.long_threshold) row = -1;
    else len = (int)n;
  }
  const IdxT* __restrict__ mycol = col + b;
  const unsigned short* __restrict__ myval = HAS_VAL ? reinterpret_cast<const unsigned short*>(p.val) + b : nullptr;
  uint32_t idx = 0, val = 0;
  if (hl < len) {
    idx = (uint32_t)mycol[hl];
    if (HAS_VAL) val = __ldg(myval + hl);
  }
  uint32_t acc[NH];
#pragma unroll
  for (int x = 0; x < NH; x++) acc[x] = 0;
  const int longest = __reduce_max_sync(0xffffffffu, len);
#pragma unroll 1
  for (int base = 0; base < longest; base += LPE) {
    uint32_t nidx = 0, nval = 0;
    if (base + LPE + hl < len) {
      nidx = (uint32_t)mycol[base + LPE + hl];
      if (HAS_VAL) nval = __ldg(myval + base + LPE + hl);
    }
    const int left = len - base;
    const int most = longest - base < LPE ? longest - base : LPE;
#pragma unroll 1
    for (int t = 0; t < most;) {
      if (most - t > 4) {
        f16_edges<8, HAS_VAL, VEC, LPE>(mat0, p.ldm, idx, val, t, left, cvalid, acc);
        t += 8;
      } else {
        f16_edges<4, HAS_VAL, VEC, LPE>(mat0, p.ldm, idx, val, t, left, cvalid, acc);
        t += 4;
      }
    }
    idx = nidx;
    val = nval;
  }
  if (row >= 0 && cvalid) {
    if (p.mean) {
      const float dv = rh((float)(len > 0 ? len : 1));   // (scalar_t)count, reducer.cuh:75-76
#pragma unroll
      for (int x = 0; x < NH; x++) acc[x] = h2_mean(acc[x], dv);
    }
    if (p.bias != nullptr) {
      float* dst = static_cast<float*>(p.out) + row * p.K + c;
      float v[2 * NH];
#pragma unroll
      for (int x = 0; x < 2 * NH; x++) {
        v[x] = __half2float(__ushort_as_half((unsigned short)(acc[x / 2] >> (x & 1) * 16)));
        if (c + x < p.K) v[x] = __fadd_rn(v[x], __ldg(p.bias + c + x));
      }
      if (VEC == 8 && p.K % 8 == 0) {
        reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2 % (2 * NH)], v[3 % (2 * NH)]);
        reinterpret_cast<float4*>(dst)[1] = make_float4(v[4 % (2 * NH)], v[5 % (2 * NH)], v[6 % (2 * NH)], v[7 % (2 * NH)]);
      } else {
#pragma unroll
        for (int x = 0; x < (VEC == 8 ? 8 : 1); x++)
          if (c + x < p.K) dst[x] = v[x % (2 * NH)];
      }
    } else if (VEC == 8) {
      __half* dst = static_cast<__half*>(p.out) + row * p.K + c;
      if (p.K % 8 == 0) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(acc[0], acc[NH > 1 ? 1 : 0], acc[NH > 2 ? 2 : 0], acc[NH > 3 ? 3 : 0]);
      } else {
#pragma unroll
        for (int x = 0; x < 8; x++)
          if (c + x < p.K) dst[x] = __ushort_as_half((unsigned short)(acc[x / 2 < NH ? x / 2 : 0] >> (x & 1) * 16));
      }
    } else {
      static_cast<__half*>(p.out)[row * p.K + c] = __ushort_as_half((unsigned short)acc[0]);
    }
  }
  // The rows may start before the long rows' kernel in front of them has finished (they touch nothing of it); the
  // grid as a whole ends after it.
  if (p.n_long > 0 && blockIdx.x == 0 && blockIdx.y == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

// One long row and 64 of its columns by two warps.  The first gathers chunks of 64 edges into a ring, the second adds
// them up (lane = two adjacent columns): with both in one warp an edge cost 8.6 instructions of the warp that owns the
// chain, 24 cycles, against 4.5 for the add itself (a row of 10,637 edges: 145 us, now 95).  `bar`: kHubChunks "full" and kHubChunks "empty" hardware barriers;
// both warps pass every one of them once per chunk.
template <typename IdxT, bool HAS_VAL>
__device__ void f16_hub_gather(const SpmmF16Params& p, long long row, long long c0, uint32_t ring, uint32_t* s_val, int bar) {
  const int lane = threadIdx.x & 31;
  const IdxT* __restrict__ rowptr = static_cast<const IdxT*>(p.rowptr);
  const IdxT* __restrict__ col = static_cast<const IdxT*>(p.col);
  const long long begin = (long long)rowptr[row], end = (long long)rowptr[row + 1];
  const int chunks = (int)((end - begin + 63) / 64);
  const int piece = lane & 7;
  const bool pvalid = c0 + piece * 8 < p.K;     // a piece past K lies past the pitch as well (the pitch is K rounded up to 8)
  const __half* __restrict__ src0 = p.mat + c0 + piece * 8;

  // the indices and values of two chunks are on their way while a third is gathered
  uint32_t idx[2][2], val[2][2];
  auto fetch = [&](int k, int at) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const long long e = begin + (long long)k * 64 + h * 32 + lane;
      idx[at][h] = val[at][h] = 0;
      if (e < end) {
        idx[at][h] = (uint32_t)col[e];
        if (HAS_VAL) val[at][h] = __ldg(reinterpret_cast<const unsigned short*>(p.val) + e);
      }
    }
  };
  auto gather = [&](int k, int at) {
    const int slot = k % kHubChunks;
    if (k >= kHubChunks) bar_sync(bar + kHubChunks + slot);          // the adder has left the slot
    const long long left = end - begin - (long long)k * 64;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (HAS_VAL) s_val[slot * 64 + h * 32 + lane] = h2_both(val[at][h]);
      const uint32_t dst = ring + slot * 8192 + h * 4096 + lane * 16;
      const __half* src[8];
#pragma unroll
      for (int j = 0; j < 8; j++)
        src[j] = src0 + (unsigned long long)__shfl_sync(0xffffffffu, idx[at][h], j * 4 + (lane >> 3)) * (unsigned long long)p.ldm;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (h * 32 + j * 4 + (lane >> 3) < left && pvalid) cp_async16(dst + j * 512, src[j]);
    }
    fetch(k + 2, at);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (k >= kHubChunks - 1) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kHubChunks - 1) : "memory");
      bar_arrive(bar + (k - (kHubChunks - 1)) % kHubChunks);
    }
  };
  fetch(0, 0);
  fetch(1, 1);
#pragma unroll 1
  for (int k = 0; k < chunks; k += 2) {
    gather(k, 0);
    if (k + 1 < chunks) gather(k + 1, 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int k = chunks < kHubChunks - 1 ? 0 : chunks - (kHubChunks - 1); k < chunks; k++) bar_arrive(bar + k % kHubChunks);
}

template <typename IdxT, bool HAS_VAL>
__device__ void f16_hub_add(const SpmmF16Params& p, long long row, long long c0, const char* ring, const uint32_t* s_val, int bar) {
  const int lane = threadIdx.x & 31;
  const IdxT* __restrict__ rowptr = static_cast<const IdxT*>(p.rowptr);
  const long long begin = (long long)rowptr[row], end = (long long)rowptr[row + 1];
  const int chunks = (int)((end - begin + 63) / 64);
  uint32_t acc = 0;
#pragma unroll 1
  for (int k = 0; k < chunks; k++) {
    const int slot = k % kHubChunks;
    bar_sync(bar + slot);
    const char* m = ring + slot * 8192 + lane * 4;
    const uint32_t* w = s_val + slot * 64;
    const long long left = end - begin - (long long)k * 64;
    if (left >= 64) {
      // groups of eight, the next group's operands on their way while the current one's adds run
      uint32_t x[2][8], v[2][8];
      auto load = [&](int g, int at) {
#pragma unroll
        for (int j = 0; j < 8; j++) x[at][j] = *reinterpret_cast<const uint32_t*>(m + (g * 8 + j) * 128);
        if (HAS_VAL) {
          const uint4 p0 = *reinterpret_cast<const uint4*>(w + g * 8), p1 = *reinterpret_cast<const uint4*>(w + g * 8 + 4);
          v[at][0] = p0.x; v[at][1] = p0.y; v[at][2] = p0.z; v[at][3] = p0.w;
          v[at][4] = p1.x; v[at][5] = p1.y; v[at][6] = p1.z; v[at][7] = p1.w;
        }
      };
      load(0, 0);
#pragma unroll
      for (int g = 0; g < 8; g++) {
        if (g < 7) load(g + 1, (g + 1) & 1);
#pragma unroll
        for (int j = 0; j < 8; j++) acc = h2_add(acc, HAS_VAL ? h2_mul(v[g & 1][j], x[g & 1][j]) : x[g & 1][j]);
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < (int)left; j++) {
        const uint32_t x = *reinterpret_cast<const uint32_t*>(m + j * 128);
        acc = h2_add(acc, HAS_VAL ? h2_mul(w[j], x) : x);
      }
    }
    if (k + kHubChunks < chunks) bar_arrive(bar + kHubChunks + slot);
  }
  if (p.mean) acc = h2_mean(acc, rh((float)(end - begin > 0 ? end - begin : 1)));
  const long long c = c0 + lane * 2;
  if (p.bias != nullptr) {
    float* dst = static_cast<float*>(p.out) + row * p.K + c;
    if (c < p.K) dst[0] = __fadd_rn(__half2float(__ushort_as_half((unsigned short)acc)), __ldg(p.bias + c));
    if (c + 1 < p.K) dst[1] = __fadd_rn(__half2float(__ushort_as_half((unsigned short)(acc >> 16))), __ldg(p.bias + c + 1));
    return;
  }
  __half* dst = static_cast<__half*>(p.out) + row * p.K + c;
  if (c < p.K) dst[0] = __ushort_as_half((unsigned short)acc);
  if (c + 1 < p.K) dst[1] = __ushort_as_half((unsigned short)(acc >> 16));
}

template <typename IdxT, bool HAS_VAL>
__global__ void __launch_bounds__(kHubPairs * 64) spmm_f16_hub_kernel(const __grid_constant__ SpmmF16Params p) {
  extern __shared__ __align__(128) char smem[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int pair = threadIdx.x >> 6;
  const long long unit = (long long)blockIdx.x * kHubPairs + pair;
  if (unit >= p.hub_units) return;
  const long long blocks = (p.K + 63) / 64;
  const long long row = p.long_row[unit / blocks], c0 = unit % blocks * 64;
  char* ring = smem + pair * kHubRing;
  uint32_t* s_val = reinterpret_cast<uint32_t*>(smem + kHubPairs * kHubRing) + pair * kHubChunks * 64;
  const int bar = pair * 2 * kHubChunks;
  if (threadIdx.x & 32)
    f16_hub_add<IdxT, HAS_VAL>(p, row, c0, ring, s_val, bar);
  else
    f16_hub_gather<IdxT, HAS_VAL>(p, row, c0, (uint32_t)__cvta_generic_to_shared(ring), s_val, bar);
}

template <typename IdxT, bool HAS_VAL, int VEC, int LPE>
static int launch_f16_lpe(SpmmF16Params& p, cudaStream_t st) {
  auto* rows = spmm_f16_rows_kernel<IdxT, HAS_VAL, VEC, LPE>;
  const long long per_block = kF16Warps * (32 / LPE);
  const dim3 grid((unsigned)((p.M + per_block - 1) / per_block), (unsigned)((p.K + LPE * VEC - 1) / (LPE * VEC)));
  if (p.n_long == 0) {
    rows<<<grid, kF16Warps * 32, 0, st>>>(p);
    EXB_CUDA_OK(cudaGetLastError());
    return EXB_OK;
  }
  auto* hub = spmm_f16_hub_kernel<IdxT, HAS_VAL>;
  EXB_CUDA_OK(cudaFuncSetAttribute(hub, cudaFuncAttributeMaxDynamicSharedMemorySize, kF16Smem));
  p.hub_units = p.n_long * ((p.K + 63) / 64);
  EXB_REQUIRE(p.hub_units <= 2147483647LL, "spmm_f16: too many long rows");
  hub<<<(unsigned)((p.hub_units + kHubPairs - 1) / kHubPairs), kHubPairs * 64, kF16Smem, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kF16Warps * 32);
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  EXB_CUDA_OK(cudaLaunchKernelEx(&cfg, rows, p));
  return EXB_OK;
}

template <typename IdxT, bool HAS_VAL>
static int launch_f16(SpmmF16Params& p, cudaStream_t st) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.mat) | (p.K % 8 == 0 ? reinterpret_cast<uintptr_t>(p.out) : 0);
  if (p.ldm % 8 == 0 && p.ldm >= (p.K + 7) / 8 * 8 && a % 16 == 0) {
    // whole 16-byte pieces: 64 columns on 8 lanes, 128 on 16, 256 on 32
    if (p.K <= 64) return launch_f16_lpe<IdxT, HAS_VAL, 8, 8>(p, st);
    if (p.K <= 128) return launch_f16_lpe<IdxT, HAS_VAL, 8, 16>(p, st);
    return launch_f16_lpe<IdxT, HAS_VAL, 8, 32>(p, st);
  }
  p.n_long = 0;           // rows that 16-byte pieces do not cover: lane = column, every row walked by its group
  p.long_threshold = 0;
  return launch_f16_lpe<IdxT, HAS_VAL, 1, 32>(p, st);
}

static int spmm_f16_common(SpmmF16Params& p, int idx_bytes, int reduce, cudaStream_t st) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_f16: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  reduce &= ~EXACT_SPMM_REGROUP;
  EXB_REQUIRE(reduce == EXACT_REDUCE_SUM || reduce == EXACT_REDUCE_MEAN, "spmm_f16: reduce must be sum or mean");
  EXB_REQUIRE(p.M >= 0 && p.K >= 0, "spmm_f16: negative shape");
  if (p.M == 0 || p.K == 0) return EXB_OK;
  EXB_REQUIRE(p.rowptr && p.mat && p.out, "spmm_f16: null pointer");
  EXB_REQUIRE(p.ldm >= p.K, "spmm_f16: row pitch %lld below %lld columns", p.ldm, p.K);
  EXB_REQUIRE((p.M + 3) / 4 <= 2147483647LL && p.M < (1LL << 32), "spmm_f16: too many rows");
  EXB_REQUIRE((p.K + 31) / 32 <= 65535, "spmm_f16: K too large");
  p.mean = reduce == EXACT_REDUCE_MEAN;
  if (idx_bytes == 4) return p.val ? launch_f16<int32_t, true>(p, st) : launch_f16<int32_t, false>(p, st);
  return p.val ? launch_f16<int64_t, true>(p, st) : launch_f16<int64_t, false>(p, st);
}

}  // namespace exb

using namespace exb;

extern "C" {

int exact_spmm_f16(const void* rowptr, const void* col, int idx_bytes, const void* value, const void* mat, int64_t M,
                   int64_t K, int reduce, void* out, void* stream) {
  return exact_spmm_f16_planned(rowptr, col, idx_bytes, value, mat, K, M, K, reduce, nullptr, 0, nullptr, 0, nullptr, out, stream);
}

int exact_spmm_f16_planned(const void* rowptr, const void* col, int idx_bytes, const void* value, const void* mat,
                           int64_t ldm, int64_t M, int64_t K, int reduce, const int32_t* row_order,
                           int64_t long_threshold, const int32_t* long_row, int64_t n_long, const float* bias, void* out,
                           void* stream) {
  EXB_REQUIRE(n_long >= 0 && (n_long == 0 || (long_row && long_threshold > 0)), "spmm_f16: null plan array");
  SpmmF16Params p{};
  p.rowptr = rowptr; p.col = col; p.val = static_cast<const __half*>(value); p.mat = static_cast<const __half*>(mat);
  p.out = out; p.bias = bias; p.M = M; p.K = K; p.ldm = ldm;
  p.row_order = row_order; p.long_row = long_row; p.n_long = n_long;
  p.long_threshold = n_long > 0 ? long_threshold : 0;
  return spmm_f16_common(p, idx_bytes, reduce, (cudaStream_t)stream);
}

}  // extern "C"

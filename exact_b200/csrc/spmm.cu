// CSR x dense SpMM (sum / mean), the aggregation of the quantised GCN / GraphSAGE layers.
//
// Replaces spmm.spmm_sum_fw / spmm_mean_fw and, on the transposed structure, the dense-operand
// gradient of spmm_sum_bw / spmm_mean_bw (exact/exact/cpp_extension/spmm.cc:31-139; kernel
// spmm_cuda.cu:27-104; reducer.cuh:43-85).
//
// One warp owns one output row and a tile of 32*KVT*VEC columns.  Column indices and edge values are
// fetched 32 at a time with one coalesced load and staged in shared memory; every lane then walks
// the staged list and gathers VEC-wide (128-bit when K % 4 == 0) slices of the neighbour rows, sixteen
// edges in flight at a time.  Edges are accumulated in CSR order with one FMA (or add) per edge and
// element, which is the reference's summation order (spmm_cuda.cu:86-93), so rows handled this way
// are bit-identical to it.
//
// Power-law graphs have rows with 10^4..10^5 edges; a single warp walking such a row is the whole
// kernel's critical path.  Rows longer than a threshold are therefore left out of the row kernel and
// cut into items of at most `threshold` edges; one warp per item writes a partial sum to caller-owned
// scratch, and a last small kernel adds each long row's partials in order.  Only those rows differ
// from the reference's summation order (by regrouping, within fp32 rounding).
#include <mutex>
#include <type_traits>

#include "common.cuh"

#include "exact_b200.h"

namespace exb {

struct SpmmParams {
  const void* rowptr;
  const void* col;
  const float* val;
  const float* mat;
  float* out;
  const float* bias;   // [K] added to every row of the result, or null
  long long M, K;
  long long Kout;      // columns of the result: K, or up to three fewer when the operand's rows are padded to 16-byte pieces
  int mean;
  int regroup;   // the caller accepts a regrouped per-row sum (EXACT_SPMM_REGROUP)
  long long long_threshold;  // rows with more edges are skipped by the row kernel (0: none)
  // long-row items
  const int* item_row;
  const long long* item_begin;
  const long long* item_end;
  const int* item_slot;      // scratch slot of each listed piece, or null (slot = position)
  long long n_items;
  const int* long_row;
  const int* long_item_ptr;
  long long n_long;
  float* scratch;      // [n_items, K]
  // Routed output (feature-parallel aggregation): row r is written to columns route_col0 .. + K - 1 of row
  // r % route_shard of the [route_shard, route_ld] matrix at route_dst[r / route_shard], which may be another
  // GPU's memory (plain stores).  route_n == 0: the rows go to `out`.
  float* route_dst[8];
  int route_n;
  const int* row_order;  // narrow operands: the order in which the rows are taken (a permutation), or null
  long long route_shard, route_ld, route_col0;
};

__device__ __forceinline__ float* output_row(const SpmmParams& p, long long row) {
  if (p.route_n == 0) return p.out + row * p.Kout;
  const long long owner = row / p.route_shard;
  return p.route_dst[owner] + (row - owner * p.route_shard) * p.route_ld + p.route_col0;
}

constexpr int kSpmmWarps = 4;
constexpr int kRowWarps = 8, kRowBlocks = 4, kRowBatch = 8;   // persistent row kernel: warps per block, blocks per SM, gathers in flight
constexpr int kEdgeUnroll = 16;   // gathers in flight per lane (16 against 8: 3 % faster at 128 M edges x 256 columns)

template <int VEC>
__device__ __forceinline__ void ldg_vec(const float* p, float (&o)[VEC]);
template <>
__device__ __forceinline__ void ldg_vec<4>(const float* p, float (&o)[4]) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
template <>
__device__ __forceinline__ void ldg_vec<2>(const float* p, float (&o)[2]) {
  const float2 v = __ldg(reinterpret_cast<const float2*>(p));
  o[0] = v.x; o[1] = v.y;
}
template <>
__device__ __forceinline__ void ldg_vec<1>(const float* p, float (&o)[1]) { o[0] = __ldg(p); }

// Loads that see what other kernels may still have been writing when this one started.
template <int VEC>
__device__ __forceinline__ void ld_vec(const float* p, float (&o)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  } else if constexpr (VEC == 2) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  } else {
    o[0] = __ldcg(p);
  }
}

template <int VEC>
__device__ __forceinline__ void st_vec(float* p, const float (&a)[VEC]) {
  if (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1 % VEC], a[2 % VEC], a[3 % VEC]);
  else if (VEC == 2) *reinterpret_cast<float2*>(p) = make_float2(a[0], a[1 % VEC]);
  else p[0] = a[0];
}

// Columns c .. c + VEC - 1 of a row of the result, bias added.
template <int VEC>
__device__ __forceinline__ void store_row(const SpmmParams& p, long long row, long long c, const float (&acc)[VEC]) {
  float* d = output_row(p, row) + c;
  if (p.Kout == p.K) {
    float o[VEC];
#pragma unroll
    for (int x = 0; x < VEC; x++) o[x] = p.bias != nullptr ? __fadd_rn(acc[x], __ldg(p.bias + c + x)) : acc[x];
    st_vec<VEC>(d, o);
  } else {
#pragma unroll
    for (int x = 0; x < VEC; x++)
      if (c + x < p.Kout) d[x] = p.bias != nullptr ? __fadd_rn(acc[x], __ldg(p.bias + c + x)) : acc[x];
  }
}

// Columns c .. c + VEC - 1 of long row i: its pieces' partial sums, added in the order of the edges.  BATCH of them are on
// their way at a time: with one, a hub row's few hundred pieces were a chain of as many memory latencies.
template <typename IdxT, int VEC, int BATCH>
__device__ __forceinline__ void sum_pieces(const SpmmParams& p, long long i, long long c) {
  if (c >= p.K) return;
  const IdxT* __restrict__ rowptr = reinterpret_cast<const IdxT*>(p.rowptr);
  const long long row = p.long_row[i];
  const int s0 = p.long_item_ptr[i], s1 = p.long_item_ptr[i + 1];
  const float* src = p.scratch + (long long)s0 * p.K + c;
  float acc[VEC];
#pragma unroll
  for (int x = 0; x < VEC; x++) acc[x] = 0.f;
  for (int s = s0; s < s1; s += BATCH, src += BATCH * p.K) {
    float m[BATCH][VEC];
#pragma unroll
    for (int u = 0; u < BATCH; u++)
      if (s + u < s1) ld_vec<VEC>(src + u * p.K, m[u]);
#pragma unroll
    for (int u = 0; u < BATCH; u++)
      if (s + u < s1) {
#pragma unroll
        for (int x = 0; x < VEC; x++) acc[x] = __fadd_rn(acc[x], m[u][x]);
      }
  }
  if (p.mean) {
    const long long cnt = (long long)rowptr[row + 1] - (long long)rowptr[row];
    const float dv = (float)(cnt > 0 ? cnt : 1);
#pragma unroll
    for (int x = 0; x < VEC; x++) acc[x] = __fdiv_rn(acc[x], dv);
  }
  store_row<VEC>(p, row, c, acc);
}

// acc += sum over edges [begin, end) of val[e] * mat[col[e], column tile], in edge order.
// FULL: every lane's KVT chunks lie inside K (no column predicate in the inner loop).
template <typename IdxT, int VEC, int KVT, bool HAS_VAL, bool FULL>
__device__ __forceinline__ void accumulate_edges(const SpmmParams& p, long long begin, long long end,
                                                 const long long (&coff)[KVT], const bool (&cvalid)[KVT],
                                                 uint32_t* s_idx, float* s_val, int lane,
                                                 float (&acc)[KVT][VEC]) {
  const IdxT* __restrict__ col = reinterpret_cast<const IdxT*>(p.col);
  const unsigned long long row_bytes = (unsigned long long)p.K * 4ull;
  const char* __restrict__ mat0 = reinterpret_cast<const char*>(p.mat + coff[0]);
  for (long long base = begin; base < end; base += 32) {
    const long long e = base + lane;
    uint32_t idx = 0;
    float v = 0.f;
    if (e < end) {
      idx = (uint32_t)col[e];
      if (HAS_VAL) v = __ldg(p.val + e);
    }
    __syncwarp();
    s_idx[lane] = idx;
    if (HAS_VAL) s_val[lane] = v;
    __syncwarp();
    const int cnt = (end - base) < 32 ? (int)(end - base) : 32;
    int i = 0;
    // full groups of kEdgeUnroll edges: all gathers issued before the first add
    for (; i + kEdgeUnroll <= cnt; i += kEdgeUnroll) {
      float m[kEdgeUnroll][KVT][VEC];
      float w[kEdgeUnroll];
#pragma unroll
      for (int u = 0; u < kEdgeUnroll; u++) {
        const float* src = reinterpret_cast<const float*>(mat0 + (unsigned long long)s_idx[i + u] * row_bytes);
        if (HAS_VAL) w[u] = s_val[i + u];
#pragma unroll
        for (int j = 0; j < KVT; j++)
          if (FULL || cvalid[j]) ldg_vec<VEC>(src + j * (32 * VEC), m[u][j]);
      }
#pragma unroll
      for (int u = 0; u < kEdgeUnroll; u++) {
#pragma unroll
        for (int j = 0; j < KVT; j++) {
          if (FULL || cvalid[j]) {
#pragma unroll
            for (int x = 0; x < VEC; x++) {
              if (HAS_VAL) acc[j][x] = __fmaf_rn(w[u], m[u][j][x], acc[j][x]);
              else acc[j][x] = __fadd_rn(acc[j][x], m[u][j][x]);
            }
          }
        }
      }
    }
    // remainder, one edge at a time
    for (; i < cnt; i++) {
      const float* src = reinterpret_cast<const float*>(mat0 + (unsigned long long)s_idx[i] * row_bytes);
      const float w = HAS_VAL ? s_val[i] : 1.f;
      float m[KVT][VEC];
#pragma unroll
      for (int j = 0; j < KVT; j++)
        if (FULL || cvalid[j]) ldg_vec<VEC>(src + j * (32 * VEC), m[j]);
#pragma unroll
      for (int j = 0; j < KVT; j++) {
        if (FULL || cvalid[j]) {
#pragma unroll
          for (int x = 0; x < VEC; x++) {
            if (HAS_VAL) acc[j][x] = __fmaf_rn(w, m[j][x], acc[j][x]);
            else acc[j][x] = __fadd_rn(acc[j][x], m[j][x]);
          }
        }
      }
    }
  }
}

enum SpmmMode { MODE_ROWS = 0, MODE_ITEMS = 1 };

// MODE_ROWS: warp per row (rows longer than long_threshold are skipped when it is non-zero).
// MODE_ITEMS: warp per long-row item, partial sums to scratch.
template <typename IdxT, int VEC, int KVT, bool HAS_VAL, bool FULL, int MODE>
__global__ void __launch_bounds__(kSpmmWarps * 32) spmm_csr_kernel(const __grid_constant__ SpmmParams p) {
  __shared__ uint32_t s_idx[kSpmmWarps][32];
  __shared__ float s_val[kSpmmWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * kSpmmWarps + warp;
  const IdxT* __restrict__ rowptr = reinterpret_cast<const IdxT*>(p.rowptr);
  const long long K = p.K;
  if (MODE == MODE_ITEMS) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  else if (p.n_items > 0 && blockIdx.x == gridDim.x - 1 && blockIdx.y == 0) asm volatile("griddepcontrol.wait;" ::: "memory");

  long long coff[KVT];
  bool cvalid[KVT];
#pragma unroll
  for (int j = 0; j < KVT; j++) {
    coff[j] = ((long long)blockIdx.y * (32 * KVT) + lane + 32 * j) * VEC;
    cvalid[j] = coff[j] < K;
  }
  float acc[KVT][VEC];
#pragma unroll
  for (int j = 0; j < KVT; j++)
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[j][e] = 0.f;

  long long begin, end;
  float* dst = nullptr;
  long long count = 0;
  if (MODE == MODE_ROWS) {
    if (unit >= p.M) return;
    begin = (long long)rowptr[unit];
    end = (long long)rowptr[unit + 1];
    count = end - begin;
    if (p.long_threshold > 0 && count > p.long_threshold) return;
  } else {
    if (unit >= p.n_items) return;
    begin = p.item_begin[unit];
    end = p.item_end[unit];
    dst = p.scratch + (long long)(p.item_slot ? p.item_slot[unit] : (int)unit) * K;
  }
  // Lanes past the last column gather the row's first columns instead (an address the lanes before them read
  // anyway) and their sums are dropped: the inner loop then carries no column predicate.  With one, the
  // compiler kept all gathers of a group live at once (96 registers against 40) and an operand of 80 - 100
  // columns took 7.0 ms at 128 M edges where 128 columns take 4.5 ms.
  long long cload[KVT];
#pragma unroll
  for (int j = 0; j < KVT; j++) cload[j] = cvalid[j] ? coff[j] : (long long)j * (32 * VEC);
  accumulate_edges<IdxT, VEC, KVT, HAS_VAL, true>(p, begin, end, cload, cvalid, s_idx[warp], s_val[warp], lane, acc);

  if (MODE == MODE_ROWS && p.mean) {
    const float dv = (float)(count > 0 ? count : 1);  // reducer.cuh:75-76
#pragma unroll
    for (int j = 0; j < KVT; j++)
#pragma unroll
      for (int x = 0; x < VEC; x++) acc[j][x] = __fdiv_rn(acc[j][x], dv);
  }
#pragma unroll
  for (int j = 0; j < KVT; j++) {
    if (!FULL && !cvalid[j]) continue;
    if (MODE == MODE_ROWS) store_row<VEC>(p, unit, coff[j], acc[j]);
    else st_vec<VEC>(dst + coff[j], acc[j]);
  }
}

template <int U, int VEC, bool HAS_VAL>
__device__ __forceinline__ void row_group(const char* __restrict__ mat0, unsigned long long row_bytes, const uint32_t* idx,
                                          const float* val, float (&acc)[VEC]) {
  float m[U][VEC];
#pragma unroll
  for (int u = 0; u < U; u++) ldg_vec<VEC>(reinterpret_cast<const float*>(mat0 + (unsigned long long)idx[u] * row_bytes), m[u]);
#pragma unroll
  for (int u = 0; u < U; u++) {
    const float w = HAS_VAL ? val[u] : 1.f;
#pragma unroll
    for (int x = 0; x < VEC; x++) {
      if (HAS_VAL) acc[x] = __fmaf_rn(w, m[u][x], acc[x]);
      else acc[x] = __fadd_rn(acc[x], m[u][x]);
    }
  }
}

// Wide operands, rows in length-sorted order, by persistent warps.  With a warp per row and blocks of four rows, a graph of
// short rows was a chain of memory latencies per row (extent, indices, gathers) at 40 % occupancy, a block's slot being held
// by its longest row.  Here a warp takes every W-th row of a tile, keeps the next row's indices, the extent of the one after
// and the id of the third on their way, and gathers eight edges at a time; 64 registers, 32 warps per SM (24 with 16
// gathers: 4 - 13 % slower, 40 with 48 registers: 10 - 20 % slower).  256 columns, with the pieces of long rows: 169,343
// nodes / 2.54 M edges 335 -> 258 us, 500,000 / 6.4 M 877 -> 634, 232,965 / 23 M 1,240 -> 1,176, 2.45 M / 126 M 9,590 -> 8,800.
// Without the order the strided rows are unbalanced (426 us at 2.54 M edges): calls without one take the kernel above.
// The pieces stay with that kernel too: 256 edges each, they want its 48 warps per SM and run 20 % slower in this one.
// Tiles of 128 columns stay separate passes over the graph (all of a tile's rows before the next tile).
template <typename IdxT, int VEC, bool HAS_VAL>
__global__ void __launch_bounds__(kRowWarps * 32, kRowBlocks) spmm_rows_kernel(const __grid_constant__ SpmmParams p) {
  __shared__ uint32_t s_idx[kRowWarps][32];
  __shared__ float s_val[kRowWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const IdxT* __restrict__ rowptr = reinterpret_cast<const IdxT*>(p.rowptr);
  const IdxT* __restrict__ col = reinterpret_cast<const IdxT*>(p.col);
  const long long K = p.K;
  const unsigned long long row_bytes = (unsigned long long)K * 4ull;
  const long long stride = (long long)gridDim.x * kRowWarps;
  uint32_t* const my_idx = s_idx[warp];
  float* const my_val = s_val[warp];

  for (long long c0 = 0; c0 < K; c0 += 32 * VEC) {
    const long long coff = c0 + lane * VEC;
    const bool cvalid = coff < K;
    const long long cload = cvalid ? coff : c0;     // lanes past K gather what the first lane gathers and drop it
    const char* __restrict__ mat0 = reinterpret_cast<const char*>(p.mat + cload);
    long long u = (long long)blockIdx.x * kRowWarps + warp;
    auto row_at = [&](long long q) -> int { return q < p.M ? p.row_order[q] : -1; };
    auto extent = [&](int r, IdxT& b, IdxT& e) {
      b = e = 0;
      if (r >= 0) {
        b = rowptr[r];
        e = rowptr[r + 1];
      }
    };
    auto first_edges = [&](IdxT b, IdxT e, uint32_t& i, float& v) {
      i = 0;
      v = 0.f;
      if (b + lane < e) {
        i = (uint32_t)col[b + lane];
        if (HAS_VAL) v = __ldg(p.val + b + lane);
      }
    };
    IdxT b, e, b1, e1;
    int row = row_at(u), row1 = row_at(u + stride), row2 = row_at(u + 2 * stride);
    extent(row, b, e);
    extent(row1, b1, e1);
    uint32_t idx;
    float val;
    first_edges(b, e, idx, val);
    for (; u < p.M; u += stride) {
      __syncwarp();
      my_idx[lane] = idx;
      if (HAS_VAL) my_val[lane] = val;
      __syncwarp();
      IdxT b2, e2;
      const int row3 = row_at(u + 3 * stride);
      extent(row2, b2, e2);
      first_edges(b1, e1, idx, val);
      const long long len = (long long)(e - b);
      if (!(p.long_threshold > 0 && len > p.long_threshold)) {
        float acc[VEC];
#pragma unroll
        for (int x = 0; x < VEC; x++) acc[x] = 0.f;
        for (long long base = 0; base < len; base += 32) {
          if (base > 0) {
            const long long at = (long long)b + base + lane;
            uint32_t i = 0;
            float v = 0.f;
            if (at < (long long)e) {
              i = (uint32_t)col[at];
              if (HAS_VAL) v = __ldg(p.val + at);
            }
            __syncwarp();
            my_idx[lane] = i;
            if (HAS_VAL) my_val[lane] = v;
            __syncwarp();
          }
          const int cnt = len - base < 32 ? (int)(len - base) : 32;
          int t = 0;
#pragma unroll 1
          for (; t + kRowBatch <= cnt; t += kRowBatch) row_group<kRowBatch, VEC, HAS_VAL>(mat0, row_bytes, my_idx + t, my_val + t, acc);
          if (kRowBatch > 8 && (cnt & 8)) { row_group<8, VEC, HAS_VAL>(mat0, row_bytes, my_idx + t, my_val + t, acc); t += 8; }
          if (cnt & 4) { row_group<4, VEC, HAS_VAL>(mat0, row_bytes, my_idx + t, my_val + t, acc); t += 4; }
          if (cnt & 2) { row_group<2, VEC, HAS_VAL>(mat0, row_bytes, my_idx + t, my_val + t, acc); t += 2; }
          if (cnt & 1) row_group<1, VEC, HAS_VAL>(mat0, row_bytes, my_idx + t, my_val + t, acc);
        }
        if (p.mean) {
          const float dv = (float)(len > 0 ? len : 1);  // reducer.cuh:75-76
#pragma unroll
          for (int x = 0; x < VEC; x++) acc[x] = __fdiv_rn(acc[x], dv);
        }
        if (cvalid) store_row<VEC>(p, row, coff, acc);
      }
      b = b1; e = e1; b1 = b2; e1 = e2;
      row = row1; row1 = row2; row2 = row3;
    }
  }
  if (p.n_items > 0) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const long long tiles = (K + 32 * VEC - 1) / (32 * VEC), units = p.n_long * tiles;
    for (long long u = (long long)blockIdx.x * kRowWarps + warp; u < units; u += stride)
      sum_pieces<IdxT, VEC, 8>(p, u / tiles, (u % tiles * 32 + lane) * VEC);
  }
}

// Adds the partial sums of each long row in item order and writes the row of the output: a warp per long row and 32 * VEC columns.
template <typename IdxT, int VEC>
__global__ void __launch_bounds__(kSpmmWarps * 32) spmm_long_reduce_kernel(const __grid_constant__ SpmmParams p) {
  const long long i = (long long)blockIdx.x * kSpmmWarps + (threadIdx.x >> 5);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (i < p.n_long) sum_pieces<IdxT, VEC, 16>(p, i, ((long long)blockIdx.y * 32 + (threadIdx.x & 31)) * VEC);
}

// Narrow operands (K <= 64): a group of LPE = 4, 8 or 16 lanes (LPE x float4 = the whole row of the operand) owns
// one row of the adjacency, so a warp works on 32 / LPE rows at once and keeps that many independent chains of
// index load -> gathers in flight.  With one row per warp a narrow operand is bound by those chains, not by
// bytes: at 128 M edges a pass over 16, 32 or 64 columns took 1.8, 2.0 and 2.8 ms against 4.4 ms for 128
// columns.  A group walks its row eight edges at a time: its lanes load the eight column indices (the next
// eight are requested before the gathers of the current ones are consumed), every lane gets each index by a
// shuffle, gathers its float4 of that source row and adds the eight in edge order, so a row's sum is the
// strict CSR-order sum (the pieces of long rows are still added separately).  The groups of a warp run until
// the longest of their rows is done; callers that pass `row_order` (rows sorted by length) give every warp rows
// of equal length.
template <typename IdxT, bool HAS_VAL, int LPE>
__global__ void __launch_bounds__(kSpmmWarps * 32) spmm_csr_multi_kernel(const __grid_constant__ SpmmParams p) {
  constexpr int kRows = 32 / LPE;              // rows (or long-row pieces) per warp
  constexpr int kBatch = 8;                    // edges per step and group
  constexpr int NI = LPE >= kBatch ? 1 : kBatch / LPE;   // index registers per lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / LPE, hl = lane % LPE;
  const long long unit = ((long long)blockIdx.x * kSpmmWarps + warp) * kRows + grp;
  const IdxT* __restrict__ rowptr = reinterpret_cast<const IdxT*>(p.rowptr);
  const IdxT* __restrict__ col = reinterpret_cast<const IdxT*>(p.col);
  const long long K = p.K;
  const long long coff = ((long long)blockIdx.y * LPE + hl) * 4;
  const bool cvalid = coff < K;

  long long begin = 0, len = 0, row = 0;
  float* dst = nullptr;
  bool live = false;
  const bool is_row = unit >= p.n_items;     // the pieces of long rows come first
  if (!is_row) {
    begin = p.item_begin[unit];
    len = p.item_end[unit] - begin;
    live = true;
    dst = p.scratch + (long long)(p.item_slot ? p.item_slot[unit] : (int)unit) * K;
  } else if (unit - p.n_items < p.M) {
    row = p.row_order ? (long long)p.row_order[unit - p.n_items] : unit - p.n_items;
    begin = (long long)rowptr[row];
    len = (long long)rowptr[row + 1] - begin;
    live = !(p.long_threshold > 0 && len > p.long_threshold);
  }
  const long long count = len;
  if (!live) len = 0;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const unsigned long long row_bytes = (unsigned long long)K * 4ull;
  const char* __restrict__ mat0 = reinterpret_cast<const char*>(p.mat + (cvalid ? coff : 0));
  const IdxT* __restrict__ mycol = col + begin;
  const float* __restrict__ myval = HAS_VAL ? p.val + begin : nullptr;

  uint32_t idx[NI];
  float val[NI];
#pragma unroll
  for (int q = 0; q < NI; q++) {
    const int pos = q * LPE + hl;
    idx[q] = 0;
    val[q] = 0.f;
    if (pos < kBatch && pos < len) {
      idx[q] = (uint32_t)mycol[pos];
      if (HAS_VAL) val[q] = __ldg(myval + pos);
    }
  }
  for (long long b = 0; __any_sync(0xffffffffu, b < len); b += kBatch) {
    uint32_t nidx[NI];
    float nval[NI];
#pragma unroll
    for (int q = 0; q < NI; q++) {
      const int in_batch = q * LPE + hl;
      const long long pos = b + kBatch + in_batch;
      nidx[q] = 0;
      nval[q] = 0.f;
      if (in_batch < kBatch && pos < len) {
        nidx[q] = (uint32_t)mycol[pos];
        if (HAS_VAL) nval[q] = __ldg(myval + pos);
      }
    }
    float4 m[kBatch];
    float w[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; j++) {
      const uint32_t ij = __shfl_sync(0xffffffffu, idx[j / LPE], j % LPE, LPE);
      w[j] = HAS_VAL ? __shfl_sync(0xffffffffu, val[j / LPE], j % LPE, LPE) : 0.f;
      m[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (b + j < len && cvalid) m[j] = __ldg(reinterpret_cast<const float4*>(mat0 + (unsigned long long)ij * row_bytes));
    }
#pragma unroll
    for (int j = 0; j < kBatch; j++) {
      if (HAS_VAL) {
        acc[0] = __fmaf_rn(w[j], m[j].x, acc[0]); acc[1] = __fmaf_rn(w[j], m[j].y, acc[1]);
        acc[2] = __fmaf_rn(w[j], m[j].z, acc[2]); acc[3] = __fmaf_rn(w[j], m[j].w, acc[3]);
      } else {
        acc[0] = __fadd_rn(acc[0], m[j].x); acc[1] = __fadd_rn(acc[1], m[j].y);
        acc[2] = __fadd_rn(acc[2], m[j].z); acc[3] = __fadd_rn(acc[3], m[j].w);
      }
    }
#pragma unroll
    for (int q = 0; q < NI; q++) {
      idx[q] = nidx[q];
      val[q] = nval[q];
    }
  }
  if (is_row && p.mean) {
    const float dv = (float)(count > 0 ? count : 1);  // reducer.cuh:75-76
#pragma unroll
    for (int x = 0; x < 4; x++) acc[x] = __fdiv_rn(acc[x], dv);
  }
  if (live && cvalid) {
    if (is_row) store_row<4>(p, row, coff, acc);
    else st_vec<4>(dst + coff, acc);
  }
}

// A launch whose blocks may start before the kernel in front of it has finished (`early`: that kernel says from where on).
template <typename... Args>
static int launch_after(void (*kernel)(Args...), dim3 grid, int threads, cudaStream_t st, bool early, const SpmmParams& p) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = early ? 1 : 0;
  EXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, p));
  return EXB_OK;
}

template <typename IdxT, int VEC>
static int launch_long_reduce(const SpmmParams& p, cudaStream_t st) {
  if (p.n_items == 0) return EXB_OK;
  const dim3 grid((unsigned)((p.n_long + kSpmmWarps - 1) / kSpmmWarps), (unsigned)((p.K + 32 * VEC - 1) / (32 * VEC)));
  return launch_after(spmm_long_reduce_kernel<IdxT, VEC>, grid, kSpmmWarps * 32, st, true, p);
}

template <typename IdxT, bool HAS_VAL, int LPE>
static int launch_spmm_multi(const SpmmParams& p, cudaStream_t st) {
  const unsigned gy = (unsigned)((p.K + 4 * LPE - 1) / (4 * LPE));
  constexpr long long per_cta = (long long)kSpmmWarps * (32 / LPE);
  dim3 grid((unsigned)((p.n_items + p.M + per_cta - 1) / per_cta), gy);
  spmm_csr_multi_kernel<IdxT, HAS_VAL, LPE><<<grid, kSpmmWarps * 32, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  return launch_long_reduce<IdxT, 4>(p, st);
}

template <typename IdxT, bool HAS_VAL>
static int launch_spmm_pair(const SpmmParams& p, cudaStream_t st) {
  if (p.K <= 16) return launch_spmm_multi<IdxT, HAS_VAL, 4>(p, st);
  if (p.K <= 32) return launch_spmm_multi<IdxT, HAS_VAL, 8>(p, st);
  return launch_spmm_multi<IdxT, HAS_VAL, 16>(p, st);
}

// The pieces of long rows first; the rows' kernel does not wait for them (programmatic launch: its blocks take the places that the
// pieces' last blocks leave free) but ends after them, and the persistent one then adds the pieces up as well.  Launched one
// after the other, the three kernels each ended with a nearly empty GPU: 169,343 nodes / 2.54 M edges x 128 columns 148 us, now
// 124, x 256 263 and 228; 60,000 / 1.2 M x 256 142 and 114; 232,965 / 23 M x 256 1,185 and 1,117.
// (One persistent kernel for pieces and rows, in any mixture, costs the pieces their 48 warps per SM: 5 % faster than separate
// launches at 2.54 M edges, 10 - 25 % slower from 20 M on.)
template <typename IdxT, int VEC, int KVT, bool HAS_VAL, bool FULL>
static int launch_spmm_mode(const SpmmParams& p, cudaStream_t st) {
  const long long C = p.K / VEC;
  const unsigned gy = (unsigned)((C + 32 * KVT - 1) / (32 * KVT));
  if (p.n_items > 0) {
    dim3 grid((unsigned)((p.n_items + kSpmmWarps - 1) / kSpmmWarps), gy);
    spmm_csr_kernel<IdxT, VEC, KVT, HAS_VAL, FULL, MODE_ITEMS><<<grid, kSpmmWarps * 32, 0, st>>>(p);
    EXB_CUDA_OK(cudaGetLastError());
  }
  // From 16 rows a warp on: with fewer the rows' own latency counts, and the other kernel keeps twice the gathers in flight
  // (12,093 rows x 256 columns 66 us here, 58 there; 38,146 rows 93 and 89; 169,343 rows 241 and 276).
  if (p.row_order != nullptr && p.M < 2147483647LL && p.M >= 16LL * sm_count() * kRowBlocks * kRowWarps) {
    long long blocks = (p.M + kRowWarps - 1) / kRowWarps;
    if (blocks > sm_count() * kRowBlocks) blocks = sm_count() * kRowBlocks;
    return launch_after(spmm_rows_kernel<IdxT, VEC, HAS_VAL>, dim3((unsigned)blocks), kRowWarps * 32, st, p.n_items > 0, p);
  }
  const dim3 grid((unsigned)((p.M + kSpmmWarps - 1) / kSpmmWarps), gy);
  const int rc = launch_after(spmm_csr_kernel<IdxT, VEC, KVT, HAS_VAL, FULL, MODE_ROWS>, grid, kSpmmWarps * 32, st, p.n_items > 0, p);
  if (rc) return rc;
  return launch_long_reduce<IdxT, VEC>(p, st);
}

template <typename IdxT, int VEC, bool HAS_VAL>
static int launch_spmm_kvt(const SpmmParams& p, cudaStream_t st) {
  const long long C = p.K / VEC;
  const long long per32 = (C + 31) / 32;
  // 128-column tiles (one float4 per lane): narrower tiles keep more source rows of a large operand in L2
  // per pass over the graph and were 5 - 13 % faster than 256- or 512-column tiles at every size measured.
  (void)per32;
  const int kvt = 1;
  const bool full = C % (32 * kvt) == 0;
#define EXB_SPMM_CASE(KVT_)                                                                          \
  if (kvt == KVT_) {                                                                                 \
    return full ? launch_spmm_mode<IdxT, VEC, KVT_, HAS_VAL, true>(p, st)                            \
                : launch_spmm_mode<IdxT, VEC, KVT_, HAS_VAL, false>(p, st);                          \
  }
  EXB_SPMM_CASE(1)
#undef EXB_SPMM_CASE
  return EXB_ERR_UNSUPPORTED;
}

template <typename IdxT, bool HAS_VAL>
static int launch_spmm_vec(const SpmmParams& p, cudaStream_t st) {
  uintptr_t a = reinterpret_cast<uintptr_t>(p.mat) | (p.Kout == p.K ? reinterpret_cast<uintptr_t>(p.out) : 0);
  if (p.scratch) a |= reinterpret_cast<uintptr_t>(p.scratch);
  for (int i = 0; i < p.route_n; i++) a |= reinterpret_cast<uintptr_t>(p.route_dst[i]);
  if (p.route_n) a |= (uintptr_t)(p.route_ld * 4) | (uintptr_t)(p.route_col0 * 4);
  if (p.K <= 64 && p.K % 4 == 0 && a % 16 == 0) return launch_spmm_pair<IdxT, HAS_VAL>(p, st);
  if (p.K % 4 == 0 && a % 16 == 0) return launch_spmm_kvt<IdxT, 4, HAS_VAL>(p, st);
  if (p.K % 2 == 0 && a % 8 == 0) return launch_spmm_kvt<IdxT, 2, HAS_VAL>(p, st);
  return launch_spmm_kvt<IdxT, 1, HAS_VAL>(p, st);
}

static int spmm_common(SpmmParams& p, int idx_bytes, int reduce, cudaStream_t st) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  p.regroup = (reduce & EXACT_SPMM_REGROUP) != 0;
  reduce &= ~EXACT_SPMM_REGROUP;
  EXB_REQUIRE(reduce == EXACT_REDUCE_SUM || reduce == EXACT_REDUCE_MEAN, "spmm: reduce must be sum or mean");
  EXB_REQUIRE(p.M >= 0 && p.K >= 0, "spmm: negative shape");
  if (p.Kout == 0) p.Kout = p.K;
  if (p.M == 0 || p.K == 0) return EXB_OK;
  EXB_REQUIRE(p.rowptr && p.mat && (p.out || p.route_n > 0), "spmm: null pointer");
  EXB_REQUIRE((p.M + kSpmmWarps - 1) / kSpmmWarps <= 2147483647LL, "spmm: too many rows");
  EXB_REQUIRE(p.K * 4 < (1LL << 32), "spmm: K too large");
  // Column indices are staged as 32-bit values (also on the int64 path): operands of 2^32 rows or more are
  // out of range.  The number of operand rows is not an argument, so the bound is stated on M (square
  // adjacencies and their row shards satisfy it whenever the operand does).
  EXB_REQUIRE(p.M < (1LL << 32), "spmm: more than 2^32 - 1 rows");
  p.mean = reduce == EXACT_REDUCE_MEAN;
  if (idx_bytes == 4) {
    return p.val ? launch_spmm_vec<int32_t, true>(p, st) : launch_spmm_vec<int32_t, false>(p, st);
  }
  return p.val ? launch_spmm_vec<int64_t, true>(p, st) : launch_spmm_vec<int64_t, false>(p, st);
}

// Gradient with respect to the edge values (spmm_cuda.cu:172-209): out[e] = dot(mat[col[e], :], grad[row[e], :])
// (/ max(row length, 1) for mean).  Lane l accumulates columns l, l + 32, ... with one FMA each, then the lanes are added by
// the reference's shuffle-down tree (l + 16, + 8, ...), so the value equals the reference's bit for bit.
// A warp takes 32 consecutive edges.  Their rows of mat are gathered eight edges at a time, the row of grad stays in
// registers while the edges belong to one row, and the 32 trees are folded into one another: at each level a lane keeps the
// half of the edges its bit names and adds the other lane's value, 31 shuffles for 32 edges instead of 160 (an addition's
// operands change places, which does not change its result).  One warp per edge was bound by issue slots and latency:
// 2.5 M edges x 128 columns 402 us, 186 us this way.
template <typename IdxT>
__global__ void __launch_bounds__(128) spmm_value_bw_kernel(const IdxT* __restrict__ row, const IdxT* __restrict__ rowptr,
                                                            const IdxT* __restrict__ col, const float* __restrict__ mat,
                                                            const float* __restrict__ grad, long long E, long long K,
                                                            int mean, float* __restrict__ out) {
  constexpr int kCols = 4;    // column groups of 32 held at a time
  const int lane = threadIdx.x & 31;
  const long long e0 = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) << 5;
  if (e0 >= E) return;
  const long long last = E - 1 - e0;
  const long long mine = e0 + (lane < last ? lane : last);      // edges past the end repeat the last one
  const long long my_row = (long long)row[mine], my_col = (long long)col[mine];
  float acc[32];
#pragma unroll
  for (int u = 0; u < 32; u++) acc[u] = 0.f;
  for (long long k0 = 0; k0 < K; k0 += 32 * kCols) {
    const long long k = k0 + lane;
    long long held = -1;
    float g[kCols];
#pragma unroll
    for (int u0 = 0; u0 < 32; u0 += 8) {
      float m[8][kCols];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float* __restrict__ src = mat + __shfl_sync(0xffffffffu, my_col, u0 + u) * K;
#pragma unroll
        for (int j = 0; j < kCols; j++) m[u][j] = k + 32 * j < K ? __ldg(src + k + 32 * j) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const long long r = __shfl_sync(0xffffffffu, my_row, u0 + u);
        if (r != held) {
          held = r;
          const float* __restrict__ src = grad + r * K;
#pragma unroll
          for (int j = 0; j < kCols; j++) g[j] = k + 32 * j < K ? __ldg(src + k + 32 * j) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < kCols; j++) acc[u0 + u] = __fmaf_rn(m[u][j], g[j], acc[u0 + u]);   // (0 * 0 past the last column)
      }
    }
  }
#pragma unroll
  for (int half = 16; half > 0; half >>= 1) {
    const bool upper = (lane & half) != 0;
#pragma unroll
    for (int u = 0; u < half; u++) {
      const float keep = upper ? acc[u + half] : acc[u], give = upper ? acc[u] : acc[u + half];
      acc[u] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, half));
    }
  }
  if (lane <= last) {
    float val = acc[0];
    if (mean) {
      const long long deg = (long long)rowptr[my_row + 1] - (long long)rowptr[my_row];
      val = __fdiv_rn(val, (float)(deg > 1 ? deg : 1));
    }
    out[e0 + lane] = val;
  }
}

// Both gradients of a weighted sum or mean in one walk of the transposed structure: for row j of it (a row of the operand) and its
// edges e to rows i of grad,
//     grad_mat[j] = sum_e w[e] * grad[i]   (edge order, one FMA an edge, as spmm_rows_kernel)
//     grad_value[perm[e]] = dot(mat[j], grad[i])   (/ max(length of row i, 1) for mean; as spmm_value_bw_kernel, bit for bit:
//                           lane l takes columns l, l + 32, ..., the lanes are added by the same tree)
// A row of grad is gathered once for both and the row of mat stays in registers, where the separate kernels gathered a row per edge
// each.  Bound by the gathers' latency: persistent warps take pieces of long rows, then rows, longest first, as spmm_rows_kernel
// does, eight edges in flight.  The eight dots of a step are folded together (9 shuffles).
// 169,343 nodes / 2.2 M edges x 128 columns: 158 + 115 us in two walks, now 224.  (The next eight gathers before the dots are folded
// need registers that spill: 356 us.)
struct WeightedBwParams {
  SpmmParams s;            // the transposed structure, its weights, mat = grad, out = grad_mat
  const void* perm;        // [nnz] position of the transposed structure's edges in the forward one
  const void* fw_rowptr;   // forward rows, for mean, or null
  const float* x;          // [M, K] the operand
  float* grad_value;
};

template <int B>
__device__ __forceinline__ float fold_dots(float (&d)[B], int lane) {
  int h = 16;
#pragma unroll
  for (int n = B; n > 1; n >>= 1, h >>= 1) {
    const bool upper = (lane & h) != 0;
#pragma unroll
    for (int u = 0; u < n / 2; u++)
      d[u] = __fadd_rn(upper ? d[u + n / 2] : d[u], __shfl_xor_sync(0xffffffffu, upper ? d[u] : d[u + n / 2], h));
  }
#pragma unroll
  for (; h > 0; h >>= 1) d[0] = __fadd_rn(d[0], __shfl_xor_sync(0xffffffffu, d[0], h));
  return d[0];
}

// What a lane needs of the matrices: grad0 / grad_last at its first and last column (lanes past K: a column of the row, dropped).
struct WeightedBwLane {
  const float* g0;
  const float* g_last;
  unsigned long long K;
  bool last_valid;
  int lane;
};

template <int B, int NC>
__device__ __forceinline__ void weighted_bw_load(const WeightedBwLane& l, const uint32_t* idx, float (&m)[B][NC]) {
#pragma unroll
  for (int u = 0; u < B; u++) {
    const unsigned long long at = (unsigned long long)idx[u] * l.K;
#pragma unroll
    for (int c = 0; c < NC - 1; c++) m[u][c] = __ldg(l.g0 + at + 32 * c);
    m[u][NC - 1] = __ldg(l.g_last + at);
  }
}

template <int B, int NC>
__device__ __forceinline__ void weighted_bw_add(const WeightedBwLane& l, const float* val, float (&m)[B][NC], const float (&xr)[NC],
                                                float (&acc)[NC], float (&d)[B]) {
#pragma unroll
  for (int u = 0; u < B; u++) {
    const float w = val[u];
    if (!l.last_valid) m[u][NC - 1] = 0.f;
    d[u] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; c++) {
      d[u] = __fmaf_rn(xr[c], m[u][c], d[u]);
      acc[c] = __fmaf_rn(w, m[u][c], acc[c]);
    }
  }
}

template <int B, typename IdxT>
__device__ __forceinline__ void weighted_bw_values(const WeightedBwParams& p, const uint32_t* idx, const IdxT* perm, int lane, float (&d)[B]) {
  float v = fold_dots<B>(d, lane);
  constexpr int kLanes = 32 / B;                // the edge of lane l is l / kLanes
  if (lane % kLanes == 0) {
    const int e = lane / kLanes;
    if (p.fw_rowptr) {
      const IdxT* rp = static_cast<const IdxT*>(p.fw_rowptr) + idx[e];
      const long long deg = (long long)rp[1] - (long long)rp[0];
      v = __fdiv_rn(v, (float)(deg > 1 ? deg : 1));
    }
    p.grad_value[perm[e]] = v;
  }
}

template <typename IdxT, int NC>
__global__ void __launch_bounds__(kRowWarps * 32, NC <= 4 ? 3 : 2) spmm_weighted_bw_kernel(const __grid_constant__ WeightedBwParams p) {
  __shared__ uint32_t s_idx[kRowWarps][32];
  __shared__ float s_val[kRowWarps][32];
  __shared__ IdxT s_perm[kRowWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const IdxT* __restrict__ rowptr = static_cast<const IdxT*>(p.s.rowptr);
  const IdxT* __restrict__ col = static_cast<const IdxT*>(p.s.col);
  const IdxT* __restrict__ perm = static_cast<const IdxT*>(p.perm);
  const long long K = p.s.K, units = p.s.n_items + p.s.M, stride = (long long)gridDim.x * kRowWarps;
  const int last = 32 * (NC - 1) + lane;
  const bool last_valid = last < K;
  const WeightedBwLane l{p.s.mat + lane, p.s.mat + (last_valid ? last : 32 * (NC - 1)), (unsigned long long)K, last_valid, lane};
  uint32_t* const my_idx = s_idx[warp];
  float* const my_val = s_val[warp];
  IdxT* const my_perm = s_perm[warp];

  struct Unit {
    long long row, slot;     // slot: of a piece, -1 for a row
    IdxT b, e;
  };
  auto unit_at = [&](long long q) {
    Unit u{0, -1, 0, 0};
    if (q < p.s.n_items) {
      u.row = p.s.item_row[q];
      u.slot = p.s.item_slot ? p.s.item_slot[q] : q;
      u.b = (IdxT)p.s.item_begin[q];
      u.e = (IdxT)p.s.item_end[q];
    } else if (q < units) {
      u.row = p.s.row_order ? (long long)p.s.row_order[q - p.s.n_items] : q - p.s.n_items;
      u.b = rowptr[u.row];
      u.e = rowptr[u.row + 1];
    }
    return u;
  };
  uint32_t idx;
  float val;
  IdxT pos;
  auto edges = [&](long long at, long long end) {
    idx = 0;
    val = 0.f;
    pos = 0;
    if (at < end) {
      idx = (uint32_t)col[at];
      val = __ldg(p.s.val + at);
      pos = perm[at];
    }
  };
  long long q = (long long)blockIdx.x * kRowWarps + warp;
  Unit cur = unit_at(q), nxt = unit_at(q + stride);
  edges((long long)cur.b + lane, (long long)cur.e);
  for (; q < units; q += stride) {
    const long long len = (long long)(cur.e - cur.b);
    const bool skip = cur.slot < 0 && p.s.long_threshold > 0 && len > p.s.long_threshold;   // done by its pieces
    const Unit after = unit_at(q + 2 * stride);
    float xr[NC], acc[NC];
    if (!skip) {
      const float* __restrict__ x = p.x + cur.row * K;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        acc[c] = 0.f;
        xr[c] = c < NC - 1 || last_valid ? __ldg(x + lane + 32 * c) : 0.f;
      }
    }
    for (long long base = 0; base == 0 || (base < len && !skip); base += 32) {
      __syncwarp();
      my_idx[lane] = idx;
      my_val[lane] = val;
      my_perm[lane] = pos;
      __syncwarp();
      // the next edges of this unit, or the first ones of the next
      if (!skip && base + 32 < len) edges((long long)cur.b + base + 32 + lane, (long long)cur.e);
      else edges((long long)nxt.b + lane, (long long)nxt.e);
      if (skip) break;
      const int cnt = len - base < 32 ? (int)(len - base) : 32;
      int t = 0;
      auto few = [&](auto n) {
        constexpr int B = decltype(n)::value;
        float m[B][NC], d[B];
        weighted_bw_load<B, NC>(l, my_idx + t, m);
        weighted_bw_add<B, NC>(l, my_val + t, m, xr, acc, d);
        weighted_bw_values<B, IdxT>(p, my_idx + t, my_perm + t, lane, d);
        t += B;
      };
#pragma unroll 1
      while (t + 8 <= cnt) few(std::integral_constant<int, 8>());
      if (cnt & 4) few(std::integral_constant<int, 4>());
      if (cnt & 2) few(std::integral_constant<int, 2>());
      if (cnt & 1) few(std::integral_constant<int, 1>());
    }
    if (!skip) {
      float* dst = cur.slot >= 0 ? p.s.scratch + cur.slot * K : p.s.out + cur.row * K;
#pragma unroll
      for (int c = 0; c < NC; c++)
        if (c < NC - 1 || last_valid) dst[lane + 32 * c] = acc[c];
    }
    cur = nxt;
    nxt = after;
  }
}

// No columns: the dots are empty sums.
template <typename IdxT>
__global__ void __launch_bounds__(256) zero_edge_values_kernel(const IdxT* __restrict__ rowptr, long long M, float* __restrict__ out) {
  const long long nnz = (long long)rowptr[M];
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < nnz; e += (long long)gridDim.x * 256) out[e] = 0.f;
}

template <typename IdxT>
static int launch_weighted_bw(const WeightedBwParams& p, cudaStream_t st) {
  const int nc = (int)((p.s.K + 31) / 32);
#define EXB_WBW(NC_)                                                                                                       \
  case NC_: {                                                                                                              \
    const int grid = resident_blocks<spmm_weighted_bw_kernel<IdxT, NC_>>(kRowWarps * 32, (p.s.n_items + p.s.M + kRowWarps - 1) / kRowWarps); \
    spmm_weighted_bw_kernel<IdxT, NC_><<<grid, kRowWarps * 32, 0, st>>>(p);                                                \
    break;                                                                                                                 \
  }
  switch (nc) {
    EXB_WBW(1) EXB_WBW(2) EXB_WBW(3) EXB_WBW(4) EXB_WBW(5) EXB_WBW(6) EXB_WBW(7) EXB_WBW(8)
    default: return fail(EXB_ERR_UNSUPPORTED, "spmm_weighted_backward: more than 256 columns");
  }
#undef EXB_WBW
  EXB_CUDA_OK(cudaGetLastError());
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.s.out) | reinterpret_cast<uintptr_t>(p.s.scratch);
  return p.s.K % 4 == 0 && a % 16 == 0 ? launch_long_reduce<IdxT, 4>(p.s, st) : launch_long_reduce<IdxT, 1>(p.s, st);
}

// max / min aggregation with the position of the winning edge (spmm_cuda.cu:27-104 with REDUCE = MAX / MIN;
// reducer.cuh:43-85): out[r, c] = max_e value[e] * mat[col[e], c], arg[r, c] = the first edge that attains it
// (a later edge replaces the current one only when strictly greater / smaller), rows without edges give 0 and
// arg = nnz.  One warp per row and 32 * VEC columns, edges in CSR order, eight gathers in flight; rows above the plan's
// threshold are cut into pieces (warps of their own, best value and position to scratch) that a last kernel compares in
// order, which picks the same edge.  With one gather at a time and no pieces 2.5 M edges x 128 columns took 2,270 us, now
// 259 (the gradient 500 us as a chain of tensor ops, 125 us below).
struct MinMaxParams {
  const void* rowptr;
  const void* col;
  const float* val;
  const float* mat;
  float* out;
  void* arg;
  long long M, K, nnz, long_threshold, n_items, n_long;
  const long long* item_begin;
  const long long* item_end;
  const int* item_slot;
  const int* long_row;
  const int* long_item_ptr;
  float* best;          // [n_items, K]
  long long* best_arg;  // [n_items, K]
};

template <typename IdxT, int VEC, bool HAS_VAL, bool IS_MAX>
__global__ void __launch_bounds__(128) spmm_minmax_kernel(const __grid_constant__ MinMaxParams p) {
  constexpr int kBatch = 8;
  const int lane = threadIdx.x & 31;
  const long long unit = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;   // pieces of long rows first
  const IdxT* __restrict__ rowptr = static_cast<const IdxT*>(p.rowptr);
  const IdxT* __restrict__ col = static_cast<const IdxT*>(p.col);
  const long long coff = ((long long)blockIdx.y * 32 + lane) * VEC;
  const bool cvalid = coff < p.K;
  const bool piece = unit < p.n_items;
  long long begin, end, row = 0;
  if (piece) {
    begin = p.item_begin[unit];
    end = p.item_end[unit];
  } else {
    row = unit - p.n_items;
    if (row >= p.M) return;
    begin = (long long)rowptr[row];
    end = (long long)rowptr[row + 1];
    if (p.long_threshold > 0 && end - begin > p.long_threshold) return;
  }
  const float* __restrict__ mat0 = p.mat + (cvalid ? coff : 0);
  float best[VEC];
  long long arg[VEC];
#pragma unroll
  for (int x = 0; x < VEC; x++) {
    best[x] = IS_MAX ? -3.402823466e+38f : 3.402823466e+38f;   // numeric_limits lowest() / max()
    arg[x] = p.nnz;
  }
  for (long long base = begin; base < end; base += 32) {
    const long long e = base + lane < end ? base + lane : end - 1;   // past the end the last edge again: never strictly better
    const long long src = (long long)col[e];
    const float w = HAS_VAL ? __ldg(p.val + e) : 1.f;
    const int cnt = end - base < 32 ? (int)(end - base) : 32;
#pragma unroll 1
    for (int t = 0; t < cnt; t += kBatch) {
      float m[kBatch][VEC];
#pragma unroll
      for (int u = 0; u < kBatch; u++) ldg_vec<VEC>(mat0 + __shfl_sync(0xffffffffu, src, t + u) * p.K, m[u]);
#pragma unroll
      for (int u = 0; u < kBatch; u++) {
        const float wu = HAS_VAL ? __shfl_sync(0xffffffffu, w, t + u) : 1.f;
#pragma unroll
        for (int x = 0; x < VEC; x++) {
          const float v = HAS_VAL ? __fmul_rn(wu, m[u][x]) : m[u][x];
          if (IS_MAX ? (v > best[x]) : (v < best[x])) {
            best[x] = v;
            arg[x] = base + t + u;
          }
        }
      }
    }
  }
  if (!cvalid) return;
  if (piece) {
    const long long at = (long long)p.item_slot[unit] * p.K + coff;
#pragma unroll
    for (int x = 0; x < VEC; x++) {
      p.best[at + x] = best[x];
      p.best_arg[at + x] = arg[x];
    }
    return;
  }
  const bool any = end > begin;                                  // reducer.cuh:78-84
  float o[VEC];
#pragma unroll
  for (int x = 0; x < VEC; x++) o[x] = any ? best[x] : 0.f;
  st_vec<VEC>(p.out + row * p.K + coff, o);
  IdxT* arg_out = static_cast<IdxT*>(p.arg) + row * p.K + coff;
#pragma unroll
  for (int x = 0; x < VEC; x++) arg_out[x] = (IdxT)arg[x];
}

template <typename IdxT, bool IS_MAX>
__global__ void __launch_bounds__(128) spmm_minmax_long_kernel(const __grid_constant__ MinMaxParams p) {
  const long long i = blockIdx.x;
  const long long row = p.long_row[i];
  const int s0 = p.long_item_ptr[i], s1 = p.long_item_ptr[i + 1];
  for (long long c = threadIdx.x; c < p.K; c += blockDim.x) {
    float best = IS_MAX ? -3.402823466e+38f : 3.402823466e+38f;
    long long arg = p.nnz;
    for (int s = s0; s < s1; s++) {
      const float v = p.best[(long long)s * p.K + c];
      if (IS_MAX ? (v > best) : (v < best)) {
        best = v;
        arg = p.best_arg[(long long)s * p.K + c];
      }
    }
    p.out[row * p.K + c] = best;
    static_cast<IdxT*>(p.arg)[row * p.K + c] = (IdxT)arg;
  }
}

template <typename IdxT, int VEC, bool HAS_VAL, bool IS_MAX>
static int launch_minmax(const MinMaxParams& p, cudaStream_t st) {
  dim3 grid((unsigned)((p.n_items + p.M + 3) / 4), (unsigned)((p.K + 32 * VEC - 1) / (32 * VEC)));
  spmm_minmax_kernel<IdxT, VEC, HAS_VAL, IS_MAX><<<grid, 128, 0, st>>>(p);
  EXB_CUDA_OK(cudaGetLastError());
  if (p.n_items > 0) {
    spmm_minmax_long_kernel<IdxT, IS_MAX><<<(unsigned)p.n_long, 128, 0, st>>>(p);
    EXB_CUDA_OK(cudaGetLastError());
  }
  return EXB_OK;
}
template <typename IdxT, bool HAS_VAL, bool IS_MAX>
static int launch_minmax_vec(const MinMaxParams& p, cudaStream_t st) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.mat) | reinterpret_cast<uintptr_t>(p.out);
  if (p.K % 4 == 0 && a % 16 == 0) return launch_minmax<IdxT, 4, HAS_VAL, IS_MAX>(p, st);
  if (p.K % 2 == 0 && a % 8 == 0) return launch_minmax<IdxT, 2, HAS_VAL, IS_MAX>(p, st);
  return launch_minmax<IdxT, 1, HAS_VAL, IS_MAX>(p, st);
}
template <typename IdxT>
static int launch_minmax_idx(const MinMaxParams& p, bool is_max, cudaStream_t st) {
  if (p.val) return is_max ? launch_minmax_vec<IdxT, true, true>(p, st) : launch_minmax_vec<IdxT, true, false>(p, st);
  return is_max ? launch_minmax_vec<IdxT, false, true>(p, st) : launch_minmax_vec<IdxT, false, false>(p, st);
}

// Gradients of the max / min aggregation, routed to the winning edges (spmm.cc:159-193, 210-241): with e = arg[r, c],
//   grad_mat[col[e], c] += value[e] * grad[r, c],   grad_value[e] += mat[col[e], c] * grad[r, c];
// rows without edges (e = nnz) contribute nothing.  One pass over arg and grad with reductions into zeroed outputs, where the
// reference's chain of tensor ops reads and writes a dozen [M, K] tensors (four of them int64).  One warp per row.
template <typename IdxT>
__global__ void __launch_bounds__(256) spmm_minmax_bw_kernel(const IdxT* __restrict__ col, const float* __restrict__ val,
                                                             const float* __restrict__ mat, const IdxT* __restrict__ arg,
                                                             const float* __restrict__ grad, long long M, long long K,
                                                             long long nnz, float* __restrict__ grad_mat,
                                                             float* __restrict__ grad_value) {
  constexpr int kBatch = 4;
  const int lane = threadIdx.x & 31;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < M; r += warps) {
    for (long long c0 = lane; c0 < K; c0 += 32 * kBatch) {
      long long e[kBatch], dst[kBatch];
      float g[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; u++) {
        const long long c = c0 + 32 * u;
        e[u] = c < K ? (long long)arg[r * K + c] : nnz;
        g[u] = c < K ? __ldg(grad + r * K + c) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kBatch; u++) dst[u] = e[u] < nnz ? (long long)col[e[u]] * K + c0 + 32 * u : -1;
#pragma unroll
      for (int u = 0; u < kBatch; u++) {
        if (dst[u] < 0) continue;
        if (grad_mat) atomicAdd(grad_mat + dst[u], val ? __fmul_rn(__ldg(val + e[u]), g[u]) : g[u]);
        if (grad_value) atomicAdd(grad_value + e[u], __fmul_rn(__ldg(mat + dst[u]), g[u]));
      }
    }
  }
}

}  // namespace exb

using namespace exb;

extern "C" {

int exact_spmm_minmax(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat,
                      int64_t M, int64_t K, int64_t nnz, int is_max, float* out, void* arg_out, void* stream) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_minmax: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  EXB_REQUIRE(M >= 0 && K >= 0 && nnz >= 0, "spmm_minmax: negative shape");
  return exact_spmm_minmax_planned(rowptr, col, idx_bytes, value, mat, M, K, nnz, is_max, 0, nullptr, nullptr, nullptr, 0, nullptr,
                                   nullptr, 0, nullptr, out, arg_out, stream);
}

int64_t exact_spmm_minmax_scratch_bytes(int64_t n_items, int64_t K) { return n_items > 0 && K > 0 ? n_items * K * 12 : 0; }

int exact_spmm_minmax_planned(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat, int64_t M,
                              int64_t K, int64_t nnz, int is_max, int64_t long_threshold, const int64_t* item_begin,
                              const int64_t* item_end, const int32_t* item_slot, int64_t n_items, const int32_t* long_row,
                              const int32_t* long_item_ptr, int64_t n_long, void* scratch, float* out, void* arg_out,
                              void* stream) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_minmax: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  EXB_REQUIRE(M >= 0 && K >= 0 && nnz >= 0, "spmm_minmax: negative shape");
  if (M == 0 || K == 0) return EXB_OK;
  EXB_REQUIRE(rowptr && mat && out && arg_out && (nnz == 0 || col), "spmm_minmax: null pointer");
  EXB_REQUIRE(n_items >= 0 && n_long >= 0 && n_items + M <= 4LL * 2147483647LL && (K + 31) / 32 <= 65535, "spmm_minmax: shape too large");
  if (n_items > 0)
    EXB_REQUIRE(long_threshold > 0 && item_begin && item_end && item_slot && long_row && long_item_ptr && scratch && n_long > 0 &&
                    (reinterpret_cast<uintptr_t>(scratch) & 7) == 0,
                "spmm_minmax: null plan array or misaligned scratch");
  MinMaxParams p{};
  p.rowptr = rowptr; p.col = col; p.val = value; p.mat = mat; p.out = out; p.arg = arg_out; p.M = M; p.K = K; p.nnz = nnz;
  p.long_threshold = n_items > 0 ? long_threshold : 0;
  p.n_items = n_items; p.n_long = n_long; p.item_begin = reinterpret_cast<const long long*>(item_begin);
  p.item_end = reinterpret_cast<const long long*>(item_end); p.item_slot = item_slot; p.long_row = long_row;
  p.long_item_ptr = long_item_ptr;
  p.best_arg = static_cast<long long*>(scratch);
  p.best = reinterpret_cast<float*>(p.best_arg + n_items * K);
  return idx_bytes == 4 ? launch_minmax_idx<int32_t>(p, is_max != 0, (cudaStream_t)stream)
                        : launch_minmax_idx<int64_t>(p, is_max != 0, (cudaStream_t)stream);
}

int exact_spmm_minmax_backward(const void* col, int idx_bytes, const float* value, const float* mat, const void* arg,
                               const float* grad_out, int64_t M, int64_t K, int64_t nnz, float* grad_mat, float* grad_value,
                               void* stream) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_minmax_backward: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  EXB_REQUIRE(M >= 0 && K >= 0 && nnz >= 0, "spmm_minmax_backward: negative shape");
  if (M == 0 || K == 0 || (!grad_mat && !grad_value)) return EXB_OK;
  EXB_REQUIRE(col && arg && grad_out && (!grad_value || mat), "spmm_minmax_backward: null pointer");
  long long blocks = (M + 7) / 8;
  if (blocks > (long long)sm_count() * 8) blocks = (long long)sm_count() * 8;
  if (idx_bytes == 4)
    spmm_minmax_bw_kernel<int32_t><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        static_cast<const int32_t*>(col), value, mat, static_cast<const int32_t*>(arg), grad_out, M, K, nnz, grad_mat, grad_value);
  else
    spmm_minmax_bw_kernel<int64_t><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        static_cast<const int64_t*>(col), value, mat, static_cast<const int64_t*>(arg), grad_out, M, K, nnz, grad_mat, grad_value);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

int exact_spmm_value_bw(const void* row, const void* rowptr, const void* col, int idx_bytes, const float* mat,
                        const float* grad, int64_t E, int64_t K, int reduce, float* out, void* stream) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_value_bw: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  EXB_REQUIRE(reduce == EXACT_REDUCE_SUM || reduce == EXACT_REDUCE_MEAN, "spmm_value_bw: reduce must be sum or mean");
  EXB_REQUIRE(E >= 0 && K >= 0, "spmm_value_bw: negative shape");
  if (E == 0) return EXB_OK;
  EXB_REQUIRE(row && col && mat && grad && out && (reduce == EXACT_REDUCE_SUM || rowptr), "spmm_value_bw: null pointer");
  EXB_REQUIRE((E + 7) / 8 <= 2147483647LL, "spmm_value_bw: too many edges");
  const unsigned blocks = (unsigned)((E + 127) / 128);   // four warps of 32 edges
  const int mean = reduce == EXACT_REDUCE_MEAN;
  if (idx_bytes == 4)
    spmm_value_bw_kernel<int32_t><<<blocks, 128, 0, (cudaStream_t)stream>>>(
        static_cast<const int32_t*>(row), static_cast<const int32_t*>(rowptr), static_cast<const int32_t*>(col), mat, grad, E,
        K, mean, out);
  else
    spmm_value_bw_kernel<int64_t><<<blocks, 128, 0, (cudaStream_t)stream>>>(
        static_cast<const int64_t*>(row), static_cast<const int64_t*>(rowptr), static_cast<const int64_t*>(col), mat, grad, E,
        K, mean, out);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

int exact_spmm_weighted_backward(const void* t_rowptr, const void* t_col, const float* t_value, const void* perm,
                                 const void* fw_rowptr, int idx_bytes, const float* mat, const float* grad, int64_t M, int64_t K,
                                 int64_t long_threshold, const int32_t* item_row, const int64_t* item_begin,
                                 const int64_t* item_end, const int32_t* item_slot, int64_t n_items, const int32_t* long_row,
                                 const int32_t* long_item_ptr, int64_t n_long, float* scratch, const int32_t* row_order,
                                 float* grad_mat, float* grad_value, void* stream) {
  EXB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, "spmm_weighted_backward: idx_bytes must be 4 or 8 (got %d)", idx_bytes);
  EXB_REQUIRE(M >= 0 && K >= 0 && n_items >= 0 && n_long >= 0, "spmm_weighted_backward: negative size");
  if (K > 256) return fail(EXB_ERR_UNSUPPORTED, "spmm_weighted_backward: more than 256 columns");
  if (M == 0) return EXB_OK;
  if (K == 0) {
    EXB_REQUIRE(t_rowptr && grad_value, "spmm_weighted_backward: null pointer");
    if (idx_bytes == 4) zero_edge_values_kernel<<<sm_count(), 256, 0, (cudaStream_t)stream>>>(static_cast<const int32_t*>(t_rowptr), M, grad_value);
    else zero_edge_values_kernel<<<sm_count(), 256, 0, (cudaStream_t)stream>>>(static_cast<const int64_t*>(t_rowptr), M, grad_value);
    EXB_CUDA_OK(cudaGetLastError());
    return EXB_OK;
  }
  EXB_REQUIRE(M < (1LL << 32) && n_items <= 2147483647LL && n_long <= 2147483647LL, "spmm_weighted_backward: too many rows");
  EXB_REQUIRE(t_rowptr && t_col && t_value && perm && mat && grad && grad_mat && grad_value, "spmm_weighted_backward: null pointer");
  if (n_items > 0)
    EXB_REQUIRE(long_threshold > 0 && item_row && item_begin && item_end && long_row && long_item_ptr && scratch && n_long > 0,
                "spmm_weighted_backward: null plan array or scratch");
  WeightedBwParams p{};
  p.s.rowptr = t_rowptr; p.s.col = t_col; p.s.val = t_value; p.s.mat = grad; p.s.out = grad_mat; p.s.M = M; p.s.K = p.s.Kout = K;
  p.s.long_threshold = n_items > 0 ? long_threshold : 0;
  p.s.item_row = item_row; p.s.item_begin = reinterpret_cast<const long long*>(item_begin);
  p.s.item_end = reinterpret_cast<const long long*>(item_end); p.s.item_slot = item_slot; p.s.n_items = n_items;
  p.s.long_row = long_row; p.s.long_item_ptr = long_item_ptr; p.s.n_long = n_long; p.s.scratch = scratch; p.s.row_order = row_order;
  p.perm = perm; p.fw_rowptr = fw_rowptr; p.x = mat; p.grad_value = grad_value;
  return idx_bytes == 4 ? launch_weighted_bw<int32_t>(p, (cudaStream_t)stream) : launch_weighted_bw<int64_t>(p, (cudaStream_t)stream);
}

int exact_spmm(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat,
               int64_t M, int64_t K, int reduce, float* out, void* stream) {
  SpmmParams p{};
  p.rowptr = rowptr; p.col = col; p.val = value; p.mat = mat; p.out = out; p.M = M; p.K = K;
  return spmm_common(p, idx_bytes, reduce, (cudaStream_t)stream);
}

int exact_spmm_split(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat,
                     int64_t M, int64_t K, int reduce, int64_t long_threshold, const int32_t* item_row,
                     const int64_t* item_begin, const int64_t* item_end, const int32_t* item_slot,
                     int64_t n_items, const int32_t* long_row, const int32_t* long_item_ptr, int64_t n_long,
                     float* scratch, float* out, void* stream) {
  EXB_REQUIRE(long_threshold > 0, "spmm_split: long_threshold must be positive");
  EXB_REQUIRE(n_items >= 0 && n_long >= 0, "spmm_split: negative plan size");
  EXB_REQUIRE(n_items <= 2147483647LL && n_long <= 2147483647LL, "spmm_split: plan too large");
  if (n_items > 0)
    EXB_REQUIRE(item_row && item_begin && item_end && long_row && long_item_ptr && scratch && n_long > 0,
                "spmm_split: null plan array or scratch");
  SpmmParams p{};
  p.rowptr = rowptr; p.col = col; p.val = value; p.mat = mat; p.out = out; p.M = M; p.K = K;
  p.long_threshold = long_threshold;
  p.item_row = item_row; p.item_begin = reinterpret_cast<const long long*>(item_begin);
  p.item_end = reinterpret_cast<const long long*>(item_end); p.item_slot = item_slot; p.n_items = n_items;
  p.long_row = long_row; p.long_item_ptr = long_item_ptr; p.n_long = n_long; p.scratch = scratch;
  return spmm_common(p, idx_bytes, reduce, (cudaStream_t)stream);
}

int exact_spmm_planned(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat, int64_t ldm,
                       int64_t M, int64_t K, int reduce, int64_t long_threshold, const int32_t* item_row, const int64_t* item_begin,
                       const int64_t* item_end, const int32_t* item_slot, int64_t n_items, const int32_t* long_row,
                       const int32_t* long_item_ptr, int64_t n_long, float* scratch, const int32_t* row_order,
                       const float* bias, float* out, void* stream) {
  EXB_REQUIRE(K >= 0 && (ldm == K || (ldm > K && ldm < K + 4 && ldm % 4 == 0)), "spmm_planned: ldm must be K, or K rounded up to a multiple of 4");
  EXB_REQUIRE(long_threshold >= 0 && n_items >= 0 && n_long >= 0, "spmm_planned: negative plan size");
  EXB_REQUIRE(n_items <= 2147483647LL && n_long <= 2147483647LL, "spmm_planned: plan too large");
  if (n_items > 0)
    EXB_REQUIRE(long_threshold > 0 && item_row && item_begin && item_end && long_row && long_item_ptr && scratch && n_long > 0,
                "spmm_planned: null plan array or scratch");
  SpmmParams p{};
  p.rowptr = rowptr; p.col = col; p.val = value; p.mat = mat; p.out = out; p.bias = bias; p.M = M; p.K = ldm; p.Kout = K;
  p.long_threshold = n_items > 0 ? long_threshold : 0;
  p.item_row = item_row; p.item_begin = reinterpret_cast<const long long*>(item_begin);
  p.item_end = reinterpret_cast<const long long*>(item_end); p.item_slot = item_slot; p.n_items = n_items;
  p.long_row = long_row; p.long_item_ptr = long_item_ptr; p.n_long = n_long; p.scratch = scratch;
  p.row_order = row_order;
  return spmm_common(p, idx_bytes, reduce, (cudaStream_t)stream);
}

int exact_spmm_split_routed(const void* rowptr, const void* col, int idx_bytes, const float* value, const float* mat,
                            int64_t M, int64_t K, int reduce, int64_t long_threshold, const int32_t* item_row,
                            const int64_t* item_begin, const int64_t* item_end, const int32_t* item_slot,
                            int64_t n_items, const int32_t* long_row, const int32_t* long_item_ptr, int64_t n_long,
                            float* scratch, const int32_t* row_order, int64_t shard, int64_t col0, int64_t ldd,
                            void* const* dst, int n_dst, void* stream) {
  EXB_REQUIRE(long_threshold >= 0 && n_items >= 0 && n_long >= 0, "spmm_split_routed: negative plan size");
  EXB_REQUIRE(n_items <= 2147483647LL && n_long <= 2147483647LL, "spmm_split_routed: plan too large");
  if (n_items > 0)
    EXB_REQUIRE(long_threshold > 0 && item_row && item_begin && item_end && long_row && long_item_ptr && scratch &&
                    n_long > 0,
                "spmm_split_routed: null plan array or scratch");
  EXB_REQUIRE(n_dst >= 1 && n_dst <= 8 && dst != nullptr, "spmm_split_routed: 1 to 8 destinations");
  EXB_REQUIRE(shard > 0 && (int64_t)n_dst * shard >= M, "spmm_split_routed: %d destinations of %lld rows do not hold %lld rows",
              n_dst, (long long)shard, (long long)M);
  EXB_REQUIRE(col0 >= 0 && K >= 0 && ldd >= col0 + K, "spmm_split_routed: columns %lld .. %lld exceed the row pitch %lld",
              (long long)col0, (long long)(col0 + K), (long long)ldd);
  SpmmParams p{};
  p.rowptr = rowptr; p.col = col; p.val = value; p.mat = mat; p.out = nullptr; p.M = M; p.K = K;
  p.long_threshold = n_items > 0 ? long_threshold : 0;
  p.item_row = item_row; p.item_begin = reinterpret_cast<const long long*>(item_begin);
  p.item_end = reinterpret_cast<const long long*>(item_end); p.item_slot = item_slot; p.n_items = n_items;
  p.long_row = long_row; p.long_item_ptr = long_item_ptr; p.n_long = n_long; p.scratch = scratch;
  p.route_n = n_dst; p.route_shard = shard; p.route_ld = ldd; p.route_col0 = col0;
  p.row_order = row_order;
  for (int i = 0; i < n_dst; i++) {
    EXB_REQUIRE(dst[i] != nullptr, "spmm_split_routed: null destination %d", i);
    p.route_dst[i] = static_cast<float*>(dst[i]);
  }
  return spmm_common(p, idx_bytes, reduce, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------------
// exact_spmm_split for callers that cannot allocate device memory: the partial sums of the long-row
// pieces live in a fixed array inside the library image instead of a caller-supplied buffer.
static __device__ __align__(256) float g_split_scratch[EXACT_SPMM_STATIC_SCRATCH_FLOATS];

// The array's name is only a host-side handle; the device address the kernels need is looked up once
// per device (with that device current) and remembered.
static int static_scratch_address(float** out) {
  static std::mutex mu;
  static float* addr[64] = {nullptr};
  int dev = 0;
  EXB_CUDA_OK(cudaGetDevice(&dev));
  EXB_REQUIRE(dev >= 0 && dev < 64, "spmm_split_static: device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    EXB_CUDA_OK(cudaGetSymbolAddress(&p, g_split_scratch));
    addr[dev] = static_cast<float*>(p);
  }
  *out = addr[dev];
  return EXB_OK;
}

int exact_spmm_split_static(const void* rowptr, const void* col, int idx_bytes, const float* value,
                            const float* mat, int64_t M, int64_t K, int reduce, int64_t long_threshold,
                            const int32_t* item_row, const int64_t* item_begin, const int64_t* item_end,
                            const int32_t* item_slot, int64_t n_items, const int32_t* long_row,
                            const int32_t* long_item_ptr, int64_t n_long, float* out, void* stream) {
  EXB_REQUIRE(n_items >= 0 && K >= 0, "spmm_split_static: negative size");
  // compared by division: n_items * K may not fit in 64 bits
  EXB_REQUIRE(K == 0 || n_items <= (int64_t)EXACT_SPMM_STATIC_SCRATCH_FLOATS / K,
              "spmm_split_static: %lld pieces x %lld columns exceed the %lld floats of the built-in scratch array; "
              "use exact_spmm_split with a caller-owned buffer",
              (long long)n_items, (long long)K, (long long)EXACT_SPMM_STATIC_SCRATCH_FLOATS);
  float* scratch = nullptr;
  int rc = static_scratch_address(&scratch);
  if (rc) return rc;
  return exact_spmm_split(rowptr, col, idx_bytes, value, mat, M, K, reduce, long_threshold, item_row, item_begin,
                          item_end, item_slot, n_items, long_row, long_item_ptr, n_long, scratch, out, stream);
}

}  // extern "C"

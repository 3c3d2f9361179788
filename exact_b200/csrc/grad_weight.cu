// Weight gradient of a quantised linear layer straight from the packed activation:
//     G[O, k] = g^T [O x N] . dequantise(packed) [N x k]
// the product grad_output.t().mm(input) of linear_backward (exact/exact/cpp_extension/backward_func.cc:87)
// with `input` still in the form qlinear.forward saved it (exact/exact/ops.py:149-154), so that the chain
// dequantize_activation -> mm of ops.py:164-169 needs neither the [N, k] fp32 activation in HBM nor a
// second pass over g.  Up to two packed activations (the two inputs of a GraphSAGE layer, which share g:
// layers.py:163-170) are multiplied in one launch; the result holds their column blocks side by side.  The
// caller applies the transposed projection to the small result: (g^T Xq) R^T.
//
// Arithmetic: as accurate as the fp32 product it replaces.  Both operands are split into an fp16 head and an fp16 tail
// (11 + 11 bits), the products head * head, head * tail and tail * head are accumulated in fp32 by tcgen05 (the fourth is below
// 2^-24).  fp16 has too few exponents for a gradient, so a stage of 64 node rows is first scaled by powers of two: each output's
// 64 gradients by their largest magnitude, the activation by a bound of its 64 rows (from their statistics).  An element keeps at
// least 2^-40 of the largest one of its 64, 2^-16 of what an fp32 sum that holds the largest one resolves (gradients all
// below 2^-100 lose digits).  The tensor core's accumulator truncates, a bias that grows with the number of steps, so a stage
// is one chain of twelve steps, the eight small products first, and its sum is taken over into fp32 registers with the
// scales undone and what the last four steps lose on average, 2^-23, given back.  Non-finite gradients make their output's row of
// G non-finite (an infinity gives NaN), non-finite activations everything their row meets, as in an fp32 product.
//
// Shape of the work.  The contraction runs over node rows, which are the slow dimension of both operands in memory, while the
// MMA wants it contiguous.  A CTA owns 128 outputs x up to 128 activation columns x a range of stages; its 28 warps:
//   warp 0       loads a [64 rows x 128 outputs] box of g by TMA and the window of packed bytes that holds the stage's rows by one bulk
//                copy, into a ring of stages;
//   warps 2-3    prepare the rows' statistics (up to 2 bits: a table of split values) and copy packed rows one by one where whole rows
//                do not fit (16-byte asynchronous copies: a bulk copy per row takes 70 cycles, longer than the products of a stage);
//   warps 4-11   A = g^T: a thread reads one output's 64 values (32 lanes read 32 consecutive words), scales and splits them and
//                writes them as its lane of tensor memory, from where the MMA takes A: the transposition costs no
//                shared-memory store and no shared-memory read of the tensor core.  Two groups of four take alternate stages;
//   warps 12-19  B = Xq: a thread dequantises part of a column (code / scale + min, as code * (1 / scale) + min) and writes heads and
//                tails as rows of K-major 128-byte-swizzled tiles;
//   warp 1       issues the MMAs: M = 128, N = the columns, K = 16;
//   warps 20-27  add an accumulator to their sums in registers, 64 columns of 32 outputs a warp, while the other one fills.
// Each of these chains is several hundred cycles of latency a stage, so each has its own warps, and short loops: with the
// statistics, B and the sums in one chain 2,449,029 x 256 outputs x (32 + 32) columns took 939 us, with A's 64 values held in registers
// (450 instructions in a row, evicting the other roles' code) 611 us, now 526 to 550; 48 outputs 265 us, 169,343 x 256 x 256 at INT2 109,
// at INT8 197, 232,965 x 256 x 602 345 us (one tf32 product: 431, 406, 101, 179 and 995).  Three quarters of the issue slots are busy.
// The CTAs that share a range of rows are neighbours in the grid, so g comes from HBM once.  Each CTA's sums go to the workspace
// and a second kernel adds them in a fixed order, so the result does not depend on timing.
//
// Every mbarrier wait is bounded; on expiry the CTA abandons its range, frees TMEM and raises the status words.
#include <cuda_fp16.h>

#include "exact_b200.h"
#include "partial_sums.cuh"
#include "tc.cuh"

namespace exb {

constexpr int kGwRows = 64;          // node rows per stage (= the K extent of a stage)
constexpr int kGwWarpsA = 4;         // warps that turn one box of g into A, in each of two groups
constexpr int kGwWarpsB = 8;
constexpr int kGwWarpsSum = 8;
constexpr int kGwThreads = (4 + 2 * kGwWarpsA + kGwWarpsB + kGwWarpsSum) * 32;
// registers a thread at launch, and after the producers of A and B have handed some to the warps that hold the sums
constexpr int kGwRegs = 72, kGwRegsA = 56, kGwRegsB = 64, kGwRegsSum = 96;
static_assert(kGwRegs + 2 * kGwRegsA + 2 * kGwRegsB + 2 * kGwRegsSum <= 7 * kGwRegs, "the registers that the block is launched with");
constexpr int kGwMaxRaw = 4;         // stages of loads, an even number; more would let the scales of B lap the sums
constexpr int kGwPrefetch = 6;       // boxes of g, and their packed rows, requested into L2 ahead of their load
constexpr int kGwASlots = 4;         // stages of A in tensor memory
constexpr int kGwBox = 128;          // outputs of a box of g; those past the last read as zero
constexpr int kGwCols = 128;         // columns of a CTA, at most
constexpr int kGwScales = 8;         // ring of the scales of A and B
constexpr int kGwPieces = 2;
// What a raw stage holds of one piece's statistics.  Up to 2 bits: for every pair of rows the heads and the tails of both rows for
// every pair of codes (8 bytes each), which a column's bytes then index: three instructions a pair of elements.  More bits: 1 / scale
// and min of every row, with which a column is dequantised and split at twelve instructions a pair.
__host__ __device__ constexpr unsigned gw_stat_bytes(int bits) {
  return bits <= 2 ? (kGwRows / 2) * (1u << (2 * bits)) * 8u : 2u * kGwRows * 4u;
}
// tensor memory: two accumulators, then the stages of A (32 columns of heads and 32 of tails each)
constexpr uint32_t kGwAcc = 128, kGwABase = 2 * kGwAcc, kGwAStage = 64, kGwTmem = 512;
static_assert(kGwABase + kGwASlots * kGwAStage <= kGwTmem, "tensor memory");

struct GwSegment {
  const uint8_t* packed;
  const uint16_t* scale_bf16;
  const uint16_t* min_bf16;
  long long pitch;           // bytes from one row of the packed stream to the next: the columns of the activation
  int c0, c1;                // its columns that this launch multiplies
  int width, tiles;          // columns of a CTA (a multiple of 16), CTAs side by side
  int part0;                 // first column of its block in the partial sums
  int window;                // a stage's packed rows come as one window, all columns of them; otherwise row by row
  unsigned long long bytes;  // of the stream; 0: not aligned to 16 bytes, read from global memory
};

struct GwParams {
  GwSegment seg[kGwPieces];
  int joint;          // both activations in one CTA (seg[0].tiles == seg[1].tiles == 1)
  int tiles;          // CTAs that share a range of rows
  float* partial;     // [splits, Opad, ldp]
  int ldp;
  int* lib_status;
  long long N, stages, per;
  int O, Opad, mtiles;
  int raw_stages;
  unsigned raw_bytes, stat_off, code_off, code_off1, code_pitch;   // one raw stage: 64 rows of g, the statistics, the packed rows
  unsigned b_tile;                                                 // bytes of a tile of B heads or tails: 128 per column
};

// What a CTA multiplies: columns c0 .. c0 + n - 1 of an activation, rows col0 .. of its B tiles.
struct GwPiece { int seg, c0, n, col0; };

// Bytes of the 16-byte pieces that hold n bytes anywhere.
__host__ __device__ inline unsigned gw_row_bytes(int n) { return (unsigned)(n + 30) & ~15u; }

__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void bulk_prefetch(const void* src, uint32_t bytes) {   // into L2; both multiples of 16
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, uint32_t bytes) {   // the rest of 16 is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// Shared memory by 32-bit address, in program order.
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float lds_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts_u4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Two values -> two fp16 heads and two fp16 tails (the first value in the lower half).
__device__ __forceinline__ void split_f16(f32x2 x, uint32_t& hi, uint32_t& lo) {
  float a, b;
  f2_unpack(x, a, b);
  const __half2 h = __floats2half2_rn(a, b);
  float d, e;      // x - head, with the head taken as it is
  asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(__half_as_ushort(__low2half(h))), "h"((uint16_t)0xbc00), "f"(a));
  asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(e) : "h"(__half_as_ushort(__high2half(h))), "h"((uint16_t)0xbc00), "f"(b));
  const __half2 l = __floats2half2_rn(d, e);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ float max_abs3(float a, float b, float c) {   // of magnitudes; three operands: an sm_100 instruction
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// The power of two that brings magnitudes up to `largest` into [2^14, 2^15), and its inverse; both normal numbers.
struct GwScale { float up, down; };
__device__ __forceinline__ GwScale gw_scale(float largest) {
  const uint32_t e = max((__float_as_uint(largest) >> 23) & 0xffu, 41u);
  return GwScale{__uint_as_float((268u - e) << 23), __uint_as_float((e - 14u) << 23)};
}

// Rows r0 .. r0 + ROWS - 1 of a stage of one column: codes out of `byte_at(q)` (packed row q of the stage), dequantised with the
// scaled statistics at `stat`, into the column's row of the head and tail tiles (row r is half-word r of 128 bytes, 16-byte chunks
// swizzled).  A block of rows is loaded before any of it is used: shared memory answers after 200 cycles here.
template <int BITS, int ROWS, class ByteAt>
__device__ __forceinline__ void gw_rows(int r0, uint32_t stat, uint32_t row, uint32_t tails, int swz, ByteAt byte_at) {
  constexpr int WPT = 8 / BITS;
  constexpr uint32_t MASK = (1u << BITS) - 1u;
  constexpr int BLOCK = BITS <= 2 ? (ROWS < 32 ? ROWS : 32) : (ROWS < 16 ? ROWS : 16);
#pragma unroll 1
  for (int rb = r0; rb < r0 + ROWS; rb += BLOCK) {
    uint32_t byte[BLOCK / WPT], hi[BLOCK / 2], lo[BLOCK / 2];
#pragma unroll
    for (int i = 0; i < BLOCK / WPT; i++) byte[i] = byte_at(rb / WPT + i);
    if constexpr (BITS <= 2) {
      constexpr uint32_t kPair = (1u << (2 * BITS)) * 8u, IDX = kPair - 8u;
      const uint32_t tab = stat + (uint32_t)(rb >> 1) * kPair;      // see gw_store_table for the places
#pragma unroll
      for (int i = 0; i < BLOCK / 2; i++) {
        const int bit = 2 * i * BITS % 8;     // of the pair's codes in their byte
        const uint32_t w = byte[2 * i * BITS / 8];
        uint32_t at = (bit >= 3 ? w >> (bit >= 3 ? bit - 3 : 0) : w << (bit < 3 ? 3 - bit : 0)) & IDX;
        if (BITS == 2) at ^= (uint32_t)(((BLOCK >= 16 ? 0 : rb >> 1) + i) & 7) * 16u;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(hi[i]), "=r"(lo[i]) : "r"(tab + i * kPair + at));
      }
    } else {
      const uint32_t inv = stat + (uint32_t)rb * 4u, mn = inv + kGwRows * 4u;
#pragma unroll
      for (int e = 0; e < BLOCK; e += 4) {
        const float4 s4 = lds_f4(inv + 4 * e), m4 = lds_f4(mn + 4 * e);
        float c[4];   // 2^23 + code
#pragma unroll
        for (int x = 0; x < 4; x++) c[x] = __uint_as_float(((byte[(e + x) / WPT] >> (((e + x) % WPT) * BITS)) & MASK) | 0x4b000000u);
        const f32x2 z = f2_pack(-8388608.f, -8388608.f);
        split_f16(f2_fma(f2_add(f2_pack(c[0], c[1]), z), f2_pack(s4.x, s4.y), f2_pack(m4.x, m4.y)), hi[e / 2], lo[e / 2]);
        split_f16(f2_fma(f2_add(f2_pack(c[2], c[3]), z), f2_pack(s4.z, s4.w), f2_pack(m4.z, m4.w)), hi[e / 2 + 1], lo[e / 2 + 1]);
      }
    }
#pragma unroll
    for (int c = 0; c < BLOCK / 8; c++) {
      const uint32_t dst = row + (uint32_t)((((rb >> 3) + c) ^ swz) << 4);
      sts_u4(dst, hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
      sts_u4(dst + tails, lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
    }
  }
}

// One lane's pair of rows 2 * lane, 2 * lane + 1 of the table that gw_rows reads: entry (code of the first) + 2^BITS * (code of the
// second), its 16-byte chunks exchanged by the pair's number at 2 bits so that eight lanes store to different banks.
template <int BITS>
__device__ __forceinline__ void gw_store_table(uint32_t stat, int lane, f32x2 inv, f32x2 mn) {
  constexpr int CODES = 1 << BITS;
  uint32_t h[CODES], l[CODES];     // of code c in both rows
#pragma unroll
  for (int c = 0; c < CODES; c++) split_f16(f2_fma(f2_pack((float)c, (float)c), inv, mn), h[c], l[c]);
#pragma unroll
  for (int e = 0; e < CODES * CODES; e += 2) {
    const int a0 = e % CODES, a1 = (e + 1) % CODES, b = e / CODES;
    const uint32_t at = (stat + (uint32_t)(lane * CODES * CODES * 8)) + (((uint32_t)e * 8u) ^ (BITS == 2 ? (uint32_t)(lane & 7) * 16u : 0u));
    sts_u4(at, __byte_perm(h[a0], h[b], 0x7610), __byte_perm(l[a0], l[b], 0x7610), __byte_perm(h[a1], h[b], 0x7610),
           __byte_perm(l[a1], l[b], 0x7610));
  }
}

template <int BITS>
__global__ void __launch_bounds__(kGwThreads, 1)
grad_weight_kernel(const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ GwParams p) {
  constexpr int WPT = 8 / BITS;
  constexpr int GROUPS = kGwRows / WPT;     // packed rows per stage
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long s_rfull[kGwMaxRaw];       // box of g, packed rows and statistics are there
  __shared__ __align__(8) unsigned long long s_rempty[kGwMaxRaw];      // ... and read
  __shared__ __align__(8) unsigned long long s_afull[kGwASlots];       // A of a stage in tensor memory
  __shared__ __align__(8) unsigned long long s_bfull[2];               // B of a stage in shared memory
  __shared__ __align__(8) unsigned long long s_done[kGwASlots];        // the MMAs of a stage have completed
  __shared__ __align__(8) unsigned long long s_drained[2];             // an accumulator has been added to the sums
  __shared__ __align__(8) unsigned long long s_scaled[kGwScales];      // the scales of a stage are in s_down and s_bdown
  __shared__ float s_down[kGwScales][128];
  __shared__ float s_bdown[kGwScales][kGwPieces];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // known to be uniform
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t b_stage = 2 * p.b_tile, raw_off = 2 * b_stage;     // the B stages first: their swizzle wants whole KB
  volatile int* abort_flag = &s_abort;
  auto wait = [&](unsigned long long& bar, uint32_t parity) {       // the same outcome in every lane
    return __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar), parity, abort_flag)) != 0;
  };

  // this CTA's part of the result
  const int tile = blockIdx.x % p.tiles, split = blockIdx.x / p.tiles;
  const int mt = tile % p.mtiles, ct = tile / p.mtiles;
  GwPiece piece0, piece1;
  int pieces = 1, part0;
  {
    const int sg = !p.joint && ct >= p.seg[0].tiles ? 1 : 0, t = ct - (sg ? p.seg[0].tiles : 0);
    const GwSegment& s = p.seg[sg];
    const int c0 = s.c0 + t * s.width;
    piece0 = GwPiece{sg, c0, min(s.width, s.c1 - c0), 0};
    part0 = s.part0 + t * s.width;
    piece1 = piece0;
    if (p.joint) {
      pieces = 2;
      piece1 = GwPiece{1, p.seg[1].c0, p.seg[1].c1 - p.seg[1].c0, s.width};
    }
  }
  const bool by_row = !p.seg[piece0.seg].window && p.seg[piece0.seg].bytes != 0;    // packed rows come one by one
  const int ncols = pieces == 2 ? piece1.col0 + (piece1.n + 15) / 16 * 16 : (piece0.n + 15) / 16 * 16;   // N of the MMAs
  const long long st0 = (long long)split * p.per;
  const long long st1 = st0 + p.per < p.stages ? st0 + p.per : p.stages;
  const int nst = st1 > st0 ? (int)(st1 - st0) : 0;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < p.raw_stages; s++) {
      mbar_init(smem_u32(&s_rfull[s]), 1 + 2 + (by_row ? 64 : 0));    // the box and windows, the statistics, the lanes that copy rows
      mbar_init(smem_u32(&s_rempty[s]), kGwWarpsA + kGwWarpsB);
    }
    for (int s = 0; s < kGwASlots; s++) {
      mbar_init(smem_u32(&s_afull[s]), kGwWarpsA);
      mbar_init(smem_u32(&s_done[s]), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(smem_u32(&s_bfull[s]), kGwWarpsB);
      mbar_init(smem_u32(&s_drained[s]), kGwWarpsSum);
    }
    for (int s = 0; s < kGwScales; s++) mbar_init(smem_u32(&s_scaled[s]), kGwWarpsA + 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(&s_tmem_base), kGwTmem);
  // rows of B that hold no column stay zero for the whole kernel
  for (uint32_t i = threadIdx.x; i < 2 * b_stage / 16; i += kGwThreads) reinterpret_cast<uint4*>(base_ptr)[i] = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;

  // A stage's packed rows of a piece begin first_of() bytes and it steps into the stream and lie in a window of 16-byte pieces.  Whole
  // windows end inside the stream up to stage whole_of() of this CTA; the one the stream ends in is copied by the warps of the
  // statistics.  (64-bit products and divisions stay out of the loops: a role is one warp's chain, five cycles an instruction.)
  const long long groups = (p.N + WPT - 1) / WPT;
  auto first_of = [&](const GwPiece& pc) { return (unsigned long long)(st0 * GROUPS) * (unsigned long long)p.seg[pc.seg].pitch; };
  auto whole_of = [&](const GwPiece& pc) {
    const GwSegment& s = p.seg[pc.seg];
    if (!s.window || s.bytes == 0) return 0;
    // first + (it + 1) * step, rounded up to 16, is at most bytes
    const unsigned long long step = (unsigned long long)GROUPS * (unsigned long long)s.pitch, end = s.bytes & ~15ull, first = first_of(pc);
    return end <= first ? 0 : (int)min((end - first) / step, (unsigned long long)nst);
  };
  // Order of the roles' progress, which the parities below rest on: A and B of stage it + 4 and it + 2 wait for the MMAs of stage it,
  // the MMAs of stage it + 2 for the sums of stage it.  So while the sums of stage it are outstanding no warp writes the scales of
  // a stage beyond it + 7, and no barrier that is waited for is more than one round ahead.
  if (warp == 0) {
    // ---------------- boxes of g, windows of packed rows ----------------
    if (lane == 0) {
      RingStage st;
      int it = 0;
      bool ok = true;
      const uint8_t *from0 = p.seg[piece0.seg].packed + first_of(piece0), *from1 = p.seg[piece1.seg].packed + first_of(piece1);
      const uint32_t step0 = (uint32_t)(GROUPS * p.seg[piece0.seg].pitch), step1 = (uint32_t)(GROUPS * p.seg[piece1.seg].pitch);
      const int whole0 = whole_of(piece0), whole1 = pieces == 2 ? whole_of(piece1) : 0;
      constexpr uint32_t box_bytes = kGwRows * kGwBox * 4;
      int row = (int)(st0 * kGwRows);
      auto window = [](const uint8_t*& from, uint32_t step) {   // its bytes; `from` moves back to its beginning
        const uint32_t skip = (uint32_t)reinterpret_cast<uintptr_t>(from) & 15u;
        from -= skip;
        return (skip + step + 15u) & ~15u;
      };
      for (; it < nst; it++, st.next(p.raw_stages)) {
        if (!mbar_wait(smem_u32(&s_rempty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
        const uint32_t full = smem_u32(&s_rfull[st.s]), dst = base + raw_off + (uint32_t)st.s * p.raw_bytes;
        const uint8_t *w0 = from0, *w1 = from1;
        const uint32_t b0 = it < whole0 ? window(w0, step0) : 0u, b1 = it < whole1 ? window(w1, step1) : 0u;
        mbar_arrive_expect_tx(full, box_bytes + b0 + b1);
        tma_load_2d(dst, &tm_g, mt * 128, row, full);
        if (b0) bulk_load(dst + p.code_off, w0, b0, full);
        if (b1) bulk_load(dst + p.code_off + p.code_off1, w1, b1, full);
        if (it + kGwPrefetch < nst) tma_prefetch_2d(&tm_g, mt * 128, row + kGwPrefetch * kGwRows);
        if (it + kGwPrefetch < whole0) {
          const uint8_t* w = from0 + kGwPrefetch * (size_t)step0;
          const uint32_t b = window(w, step0);
          bulk_prefetch(w, b);
        }
        if (it + kGwPrefetch < whole1) {
          const uint8_t* w = from1 + kGwPrefetch * (size_t)step1;
          const uint32_t b = window(w, step1);
          bulk_prefetch(w, b);
        }
        row += kGwRows;
        from0 += step0;
        from1 += step1;
      }
      if (!ok) {   // leave no copy in flight (bounded; the barrier also waits for warps that have given up as well)
        const long long t0 = clock64();
        for (int j = 0; j < p.raw_stages && j < it; j++) {
          const int jt = it - 1 - j;
          while (!mbar_try_wait(smem_u32(&s_rfull[jt % p.raw_stages]), (uint32_t)(jt / p.raw_stages) & 1u) &&
                 clock64() - t0 < kWaitLimitCycles) {}
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp walks the loop, one elected lane issues ----------------
    const bool elected = elect_one();
    const uint32_t idesc = umma_idesc_f16(128, ncols);
    int it = 0;
    for (; it < nst; it++) {
      const int a = it & (kGwASlots - 1), b = it & 1;
      if (!wait(s_drained[b], (uint32_t)((it >> 1) & 1) ^ 1u) || !wait(s_afull[a], (uint32_t)(it >> 2) & 1u) ||
          !wait(s_bfull[b], (uint32_t)(it >> 1) & 1u))
        break;
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)b * kGwAcc, ah = tmem_base + kGwABase + (uint32_t)a * kGwAStage, al = ah + 32;
      const uint64_t bh = umma_desc_sw128(base + (uint32_t)b * b_stage), bl = umma_desc_sw128(base + (uint32_t)b * b_stage + p.b_tile);
      if (elected) {
#pragma unroll
        for (int k = 0; k < kGwRows / 16; k++) {       // 16 rows: 8 columns of A, 32 bytes along the 128-byte rows of B
          umma_f16_ts(d, al + 8 * k, bh + (uint64_t)(2 * k), idesc, k != 0);
          umma_f16_ts(d, ah + 8 * k, bl + (uint64_t)(2 * k), idesc, 1);
        }
#pragma unroll
        for (int k = 0; k < kGwRows / 16; k++) umma_f16_ts(d, ah + 8 * k, bh + (uint64_t)(2 * k), idesc, 1);
        umma_commit(smem_u32(&s_done[a]));
      }
      __syncwarp();
    }
    if (it > 0) {   // no MMA under way when the tensor memory is given back, also where another role has given up (bounded)
      const long long t0 = clock64();
      while (!mbar_try_wait(smem_u32(&s_done[(it - 1) & (kGwASlots - 1)]), (uint32_t)((it - 1) >> 2) & 1u) &&
             clock64() - t0 < kWaitLimitCycles) {}
    }
  } else if (warp < 4) {
    // ---------------- statistics, and packed rows that do not come as a window ----------------
    // Warp 2 + i prepares the statistics of piece i, or of every second stage, rows 2 * lane and 2 * lane + 1 in a lane: 1 / scale (a
    // constant row has scale = inf and reciprocal 0, its codes are 0 anyway) and min, both times the stage's power of two.  Rows past N
    // get 0, 0.
    const int who = warp - 2, id = who * 32 + lane;
    const int every = pieces == 2 ? 1 : 2, lead = pieces == 2 ? 0 : who;      // its stages
    const GwPiece& mine = who && pieces == 2 ? piece1 : piece0;
    const uint16_t* scales = p.seg[mine.seg].scale_bf16 + (st0 + lead) * kGwRows + 2 * lane;
    const uint16_t* mins = p.seg[mine.seg].min_bf16 + (st0 + lead) * kGwRows + 2 * lane;
    long long rows_left = p.N - (st0 + lead) * kGwRows - 2 * lane;   // from the first of this lane's next two rows on
    uint16_t sc_next[2], mn_next[2];
    auto load_stats = [&]() {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        sc_next[h] = 0x7f80;
        mn_next[h] = 0;
        if (rows_left > h) {
          sc_next[h] = __ldg(scales + h);
          mn_next[h] = __ldg(mins + h);
        }
      }
      if (lane < 2 && rows_left > (kGwPrefetch + 1) * kGwRows)
        asm volatile("prefetch.global.L2 [%0];" ::"l"((lane ? mins : scales) + kGwPrefetch * kGwRows));
      scales += every * kGwRows;
      mins += every * kGwRows;
      rows_left -= every * kGwRows;
    };
    load_stats();
    const int mine_at = pieces == 2 ? who : 0;
    const uint32_t stat0 = base + raw_off + p.stat_off + (uint32_t)mine_at * gw_stat_bytes(BITS);
    auto store_stats = [&](int it, int place) {
      float inv[2], mn[2], largest = 0.f;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        inv[h] = __frcp_rn(bf16_bits_to_f32(sc_next[h]));
        mn[h] = bf16_bits_to_f32(mn_next[h]);
        largest = fmaxf(largest, fmaxf(fabsf(mn[h]), fabsf(__fmaf_rn((float)((1 << BITS) - 1), inv[h], mn[h]))));
      }
      load_stats();
      const GwScale sc = gw_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(largest))));   // none is negative
      const uint32_t stat = stat0 + (uint32_t)place * p.raw_bytes;
      const f32x2 up = f2_pack(sc.up, sc.up), inv2 = f2_mul(f2_pack(inv[0], inv[1]), up), mn2 = f2_mul(f2_pack(mn[0], mn[1]), up);
      if (BITS <= 2) {
        gw_store_table<BITS <= 2 ? BITS : 1>(stat, lane, inv2, mn2);
      } else {
        asm volatile("st.shared.b64 [%0], %1;" ::"r"(stat + lane * 8), "l"(inv2) : "memory");
        asm volatile("st.shared.b64 [%0], %1;" ::"r"(stat + kGwRows * 4 + lane * 8), "l"(mn2) : "memory");
      }
      if (lane == 0) s_bdown[it & (kGwScales - 1)][mine_at] = sc.down;
    };
    const int whole0 = whole_of(piece0), whole1 = pieces == 2 ? whole_of(piece1) : nst;
    const int chunks = (int)(gw_row_bytes(piece0.n) >> 4), q0 = id / chunks, k0 = id - q0 * chunks, dq = 64 / chunks, dc = 64 - dq * chunks;
    RingStage st;
    for (int it = 0; it < nst; it++, st.next(p.raw_stages)) {
      if (!wait(s_rempty[st.s], st.ph ^ 1u)) break;
      const uint32_t dst = base + raw_off + (uint32_t)st.s * p.raw_bytes + p.code_off;
      if (by_row) {
        const GwSegment& s = p.seg[piece0.seg];
        const long long grp0 = (st0 + it) * GROUPS;
        const int rows = (int)min(groups - grp0, (long long)GROUPS);
        for (int q = q0, c = k0; q < rows;) {
          const unsigned long long at = (unsigned long long)(grp0 + q) * (unsigned long long)s.pitch + piece0.c0;
          const unsigned long long from = (at & ~15ull) + 16u * (unsigned)c;
          if (from < at + piece0.n) {
            const unsigned long long rest = s.bytes - from;
            copy16(dst + (uint32_t)q * p.code_pitch + 16u * (unsigned)c, s.packed + from, rest < 16 ? (uint32_t)rest : 16u);
          }
          q += dq;
          c += dc;
          if (c >= chunks) {
            c -= chunks;
            q++;
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&s_rfull[st.s])) : "memory");
      } else if (it >= whole0 || it >= whole1) {   // the window that the stream ends in, byte by byte
        for (int i = 0; i < pieces; i++) {
          const GwPiece& pc = i ? piece1 : piece0;
          const GwSegment& s = p.seg[pc.seg];
          if (s.bytes == 0 || it < (i ? whole1 : whole0)) continue;
          const unsigned long long first = first_of(pc) + (unsigned long long)it * (unsigned long long)(GROUPS * s.pitch);
          const uint32_t skip = (uint32_t)first & 15u, n = (uint32_t)min((unsigned long long)(GROUPS * s.pitch), s.bytes - first);
          uint8_t* to = base_ptr + (dst - base) + (i ? p.code_off1 : 0u) + skip;
          for (uint32_t b = (uint32_t)id; b < n; b += 64) to[b] = __ldg(s.packed + first + b);
        }
      }
      if (pieces == 2 || (it & 1) == who) store_stats(it, st.s);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_rfull[st.s]));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < 4 + 2 * kGwWarpsA) {
    // ---------------- A = g^T, scaled and split, in tensor memory ----------------
    set_registers<kGwRegsA, false>();
    const int group = (warp - 4) / kGwWarpsA, quad = warp & 3, o = quad * 32 + lane;
    const uint32_t tlane = tmem_base + kGwABase + ((uint32_t)(quad * 32) << 16);
    RingStage st;
    if (group) st.next(p.raw_stages);
    // The ring has an even number of stages, so a group meets the same places in every round and none is a round ahead of it.
    for (int it = group; it < nst; it += 2, st.next(p.raw_stages), st.next(p.raw_stages)) {
      const int a = it & (kGwASlots - 1);
      if (!wait(s_rfull[st.s], st.ph)) break;
      // both passes read shared memory, a tenth of whose rate is in use
      const uint32_t raw = base + raw_off + (uint32_t)st.s * p.raw_bytes + (uint32_t)o * 4u;
      float m0 = 0.f, m1 = 0.f;
#pragma unroll 1
      for (uint32_t b = 0; b < kGwRows; b += 16) {
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = lds_f1(raw + b * (kGwBox * 4) + r * (kGwBox * 4));
#pragma unroll
        for (int r = 0; r < 16; r += 4) {
          m0 = max_abs3(m0, v[r], v[r + 1]);
          m1 = max_abs3(m1, v[r + 2], v[r + 3]);
        }
      }
      const GwScale sc = gw_scale(fmaxf(m0, m1));
      s_down[it & (kGwScales - 1)][o] = __uint_as_float(__float_as_uint(sc.down) + 1u);   // times 1 + 2^-23: see the top
      if (!wait(s_done[a], (uint32_t)((it >> 2) & 1) ^ 1u)) break;
      tc_fence_after();
      const uint32_t to = tlane + (uint32_t)a * kGwAStage;
      const f32x2 up = f2_pack(sc.up, sc.up);
#pragma unroll 1
      for (uint32_t b = 0; b < kGwRows; b += 16) {
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = lds_f1(raw + b * (kGwBox * 4) + r * (kGwBox * 4));
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; i++) split_f16(f2_mul(f2_pack(v[2 * i], v[2 * i + 1]), up), hi[i], lo[i]);
        tmem_st8(to + b / 2, hi);
        tmem_st8(to + 32 + b / 2, lo);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_rempty[st.s]));
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&s_scaled[it & (kGwScales - 1)]));
        mbar_arrive(smem_u32(&s_afull[a]));
      }
    }
  } else if (warp < 4 + 2 * kGwWarpsA + kGwWarpsB) {
    // ---------------- B = dequantised activation ----------------
    set_registers<kGwRegsB, false>();
    const int t = threadIdx.x - (4 + 2 * kGwWarpsA) * 32;
    // a thread owns half of a column, or a smaller share of its rows where the columns leave threads over
    const int used = pieces == 2 ? piece0.n + piece1.n : piece0.n;
    int slots = 32;
    while (slots < used) slots <<= 1;
    const int cslot = t % slots, slice = t / slots;
    const int pi = cslot >= piece0.n ? 1 : 0, j = cslot - (pi ? piece0.n : 0);
    const GwPiece pc = pi ? piece1 : piece0;
    const GwSegment& seg = p.seg[pc.seg];
    const int jb = pc.col0 + j;
    const uint32_t code_at = base + raw_off + p.code_off + (pi ? p.code_off1 : 0u) + (uint32_t)(seg.window ? pc.c0 + j : j);
    const uint32_t stat_at = base + raw_off + p.stat_off + (uint32_t)pi * gw_stat_bytes(BITS);
    // packed row q of a stage: q * stride, and the misalignment of its own where rows are copied one by one at a pitch off 16
    const uint32_t pitch = (uint32_t)seg.pitch, stride = seg.window ? pitch : p.code_pitch;
    const bool crooked = !seg.window && pitch % 16 != 0;
    uint32_t first = (uint32_t)first_of(pc) + (seg.window ? 0u : (uint32_t)pc.c0);   // of the stage's bytes; the last four bits count
    RingStage st;
    for (int it = 0; it < nst; it++, st.next(p.raw_stages), first += (uint32_t)GROUPS * pitch) {
      if (it >= 2 && !wait(s_done[(it - 2) & (kGwASlots - 1)], (uint32_t)((it - 2) >> 2) & 1u)) break;   // read by the MMAs
      if (!wait(s_rfull[st.s], st.ph)) break;
      if (cslot < used) {
        const uint32_t row = base + (uint32_t)(it & 1) * b_stage + (uint32_t)jb * 128u, stat = stat_at + (uint32_t)st.s * p.raw_bytes;
        const int swz = jb & 7;
        auto from = [&](auto byte_at) {
          switch (slots) {
            case 128: gw_rows<BITS, 32>(slice * 32, stat, row, p.b_tile, swz, byte_at); break;
            case 64: gw_rows<BITS, 16>(slice * 16, stat, row, p.b_tile, swz, byte_at); break;
            default: gw_rows<BITS, 8>(slice * 8, stat, row, p.b_tile, swz, byte_at);
          }
        };
        const uint32_t at = code_at + (uint32_t)st.s * p.raw_bytes, skip = first & 15u;
        if (seg.bytes == 0) {
          const uint8_t* src = seg.packed + (unsigned long long)((st0 + it) * GROUPS) * (unsigned long long)seg.pitch + pc.c0 + j;
          const long long left = groups - (st0 + it) * GROUPS;
          from([&](int q) { return q < left ? (uint32_t)__ldg(src + (size_t)q * seg.pitch) : 0u; });
        } else if (crooked) {
          from([&](int q) { return lds_u8(at + (uint32_t)q * stride + ((skip + (uint32_t)q * pitch) & 15u)); });
        } else {
          from([&](int q) { return lds_u8(at + skip + (uint32_t)q * stride); });
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&s_rempty[st.s]));
        mbar_arrive(smem_u32(&s_bfull[it & 1]));
        if (t == 0) mbar_arrive(smem_u32(&s_scaled[it & (kGwScales - 1)]));   // (s_bdown, seen through the ring)
      }
    }
  } else {
    // ---------------- sums ----------------
    set_registers<kGwRegsSum, true>();
    const int quad = warp & 3, half = (warp - (kGwThreads / 32 - kGwWarpsSum)) >> 2;
    float sum[64];   // columns 32 * b + 16 * half .. + 15 of output quad * 32 + lane in sum[16 * b ..]
#pragma unroll
    for (int i = 0; i < 64; i++) sum[i] = 0.f;
    const int split_col = pieces == 2 ? piece1.col0 : kGwCols;
    int it = 0;
    for (; it < nst; it++) {
      const int sl = it & (kGwScales - 1);
      if (!wait(s_scaled[sl], (uint32_t)(it >> 3) & 1u)) break;
      const float down = s_down[sl][quad * 32 + lane], down0 = down * s_bdown[sl][0], down1 = down * s_bdown[sl][pieces - 1];
      if (!wait(s_done[it & (kGwASlots - 1)], (uint32_t)(it >> 2) & 1u)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(it & 1) * kGwAcc;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int c0 = 32 * i + 16 * half;
        if (c0 < ncols) {
          float v[16];
          tmem_ld16(taddr + (uint32_t)c0, v);
          const float m = c0 < split_col ? down0 : down1;
#pragma unroll
          for (int e = 0; e < 16; e++) sum[16 * i + e] = __fmaf_rn(v[e], m, sum[16 * i + e]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_drained[it & 1]));
    }
    if (it >= nst) {   // this CTA's sums to the workspace
      float* dst = p.partial + ((size_t)split * p.Opad + mt * 128 + quad * 32 + lane) * p.ldp + part0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int c0 = 32 * i + 16 * half;
        if (c0 < ncols) {
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(dst + c0 + e) = make_float4(sum[16 * i + e], sum[16 * i + e + 1], sum[16 * i + e + 2], sum[16 * i + e + 3]);
        }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kGwTmem);
  }
  if (threadIdx.x == 0 && s_abort) raise_status(p.lib_status, EXB_STATUS_GRAD_WEIGHT);
}

// out[o, column] = sum over the row ranges, in a fixed order, of partial[split, o, column]; the columns of the second activation
// start at part1 in the sums.  In double: these last additions are few, but nothing averages their roundings.
struct GwColumns { int part1, n0, n1; long long out0, out1; };
__global__ void __launch_bounds__(32 * kSumSlices) grad_weight_reduce_kernel(const float* __restrict__ partial, int splits, int O, int Opad,
                                                                             int ldp, GwColumns c, long long ldo,
                                                                             float* __restrict__ out) {
  __shared__ double s_part[kSumSlices][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  const float a = (float)sum_partials(partial + i, (long long)Opad * ldp, splits, i < O * ldp, s_part);
  if (threadIdx.y != 0 || i >= O * ldp) return;
  const int o = i / ldp, pc = i - o * ldp, j = pc < c.part1 ? pc : pc - c.part1;
  if (j < (pc < c.part1 ? c.n0 : c.n1)) out[(size_t)o * ldo + (pc < c.part1 ? c.out0 : c.out1) + j] = a;
}

static int pad16(long long n) { return (int)((n + 15) / 16 * 16); }
static unsigned gw_window_bytes(int bits, long long pitch) { return (unsigned)(kGwRows * bits / 8 * pitch + 32 + 15) & ~15u; }

// Stages of loads that fit beside two stages of B of `cols` columns, an even number (see the producers of A).
constexpr unsigned kGwRoom = 222 * 1024;    // of the 227 KB, beside 4.5 KB of barriers and scales
static unsigned gw_raw_bytes(int bits, int pieces, unsigned code_bytes) {
  return (unsigned)(kGwRows * kGwBox * 4) + ((pieces * gw_stat_bytes(bits) + code_bytes + 127u) & ~127u);
}
static int gw_raw_stages(int cols, unsigned raw_bytes) {
  const int fit = (int)((kGwRoom - 1024 - 4u * (unsigned)cols * 128u) / raw_bytes);
  return fit >= kGwMaxRaw ? kGwMaxRaw : fit / 2 * 2;
}
// Columns a CTA takes at most: those with which four stages fit when packed rows are copied one by one (112 at INT8, else 128).
static int gw_max_cols(int bits) {
  int cols = kGwCols;
  while (cols > 16 && gw_raw_stages(cols, gw_raw_bytes(bits, 1, (unsigned)(kGwRows * bits / 8) * gw_row_bytes(cols))) < 4) cols -= 16;
  return cols;
}

// One launch: columns s0.c0 .. s0.c1 - 1 of one activation, or of two.
static int gw_launch(const float* g, int64_t N, int O, GwSegment s0, const GwSegment* s1, int bits, void* workspace,
                     int64_t workspace_bytes, float* out, int64_t ldo, int64_t out1, cudaStream_t st) {
  const int wpt = 8 / bits, groups = kGwRows / wpt, nseg = s1 ? 2 : 1, cap = gw_max_cols(bits);
  GwParams p{};
  p.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  p.lib_status = status_word_ptr();
  p.N = N; p.O = O; p.Opad = (O + 127) / 128 * 128; p.mtiles = p.Opad / 128;
  p.stages = (N + kGwRows - 1) / kGwRows;
  p.seg[0] = s0;
  if (s1) p.seg[1] = *s1;
  int cols = 0, column_tiles = 0;
  for (int i = 0; i < nseg; i++) {
    GwSegment& s = p.seg[i];
    const int n = s.c1 - s.c0;
    s.tiles = (n + cap - 1) / cap;
    s.width = pad16((n + s.tiles - 1) / s.tiles);
    s.part0 = p.ldp;
    p.ldp += s.tiles * s.width;
    column_tiles += s.tiles;
    if (s.width > cols) cols = s.width;
    s.bytes = (reinterpret_cast<uintptr_t>(s.packed) & 15) == 0
                  ? (unsigned long long)((N + wpt - 1) / wpt) * (unsigned long long)s.pitch : 0;
  }
  // Packed rows as whole windows (one bulk copy a stage) where four stages still fit, else row by row; both activations in one CTA, so
  // that g is read and split once, if both have windows.
  unsigned code_bytes = 0;
  const unsigned w0 = gw_window_bytes(bits, p.seg[0].pitch), w1 = nseg == 2 ? gw_window_bytes(bits, p.seg[1].pitch) : 0;
  if (nseg == 2 && column_tiles == 2 && p.ldp <= kGwCols && p.seg[0].pitch <= kGwCols && p.seg[1].pitch <= kGwCols &&
      gw_raw_stages(p.ldp, gw_raw_bytes(bits, 2, w0 + w1)) >= 4) {
    p.joint = 1;
    p.seg[0].window = p.seg[1].window = 1;
    p.code_off1 = w0;
    code_bytes = w0 + w1;
    cols = p.ldp;
    column_tiles = 1;
  } else {
    for (int i = 0; i < nseg; i++) {
      GwSegment& s = p.seg[i];
      const unsigned row = gw_row_bytes(s.tiles > 1 ? s.width : s.c1 - s.c0), w = i ? w1 : w0;
      if (row > p.code_pitch) p.code_pitch = row;
      s.window = s.pitch <= 4096 && gw_raw_stages(cols, gw_raw_bytes(bits, 1, w)) >= 4;
      if (s.window && w > code_bytes) code_bytes = w;
    }
    if ((!p.seg[0].window || (nseg == 2 && !p.seg[1].window)) && groups * p.code_pitch > code_bytes) code_bytes = groups * p.code_pitch;
  }
  if (s1 == nullptr) p.seg[1] = p.seg[0];
  p.b_tile = (unsigned)cols * 128u;
  p.stat_off = (unsigned)(kGwRows * kGwBox * 4);
  p.code_off = p.stat_off + (p.joint ? 2 : 1) * gw_stat_bytes(bits);
  p.raw_bytes = gw_raw_bytes(bits, p.joint ? 2 : 1, code_bytes);
  p.raw_stages = gw_raw_stages(cols, p.raw_bytes);
  EXB_REQUIRE(p.raw_stages >= 2 && p.raw_stages % 2 == 0, "grad_weight_from_packed: the pipeline does not fit in shared memory");
  p.tiles = p.mtiles * column_tiles;
  long long splits = sm_count() / p.tiles;
  if (splits > p.stages) splits = p.stages;
  if (splits < 1) splits = 1;
  p.per = (p.stages + splits - 1) / splits;
  splits = p.per > 0 ? (p.stages + p.per - 1) / p.per : 0;
  const int64_t need = 256 + (int64_t)splits * p.Opad * p.ldp * 4;
  EXB_REQUIRE(workspace_bytes >= need, "grad_weight_from_packed: workspace of %lld bytes is too small (%lld needed)",
              (long long)workspace_bytes, (long long)need);
  if (N > 0) {
    CUtensorMap tm_g;
    int rc = make_tensor_map_2d_f32(&tm_g, g, (unsigned long long)O, (unsigned long long)N, (unsigned long long)O * 4, kGwBox,
                                    kGwRows, /*swizzle128=*/false);
    if (rc) return rc;
    const size_t dyn = 1024 + 4 * (size_t)p.b_tile + (size_t)p.raw_stages * p.raw_bytes;
    auto* kern = bits == 1 ? grad_weight_kernel<1> : bits == 2 ? grad_weight_kernel<2> : bits == 4 ? grad_weight_kernel<4> : grad_weight_kernel<8>;
    EXB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    kern<<<(unsigned)(p.tiles * splits), kGwThreads, dyn, st>>>(tm_g, p);
    EXB_CUDA_OK(cudaGetLastError());
  }
  GwColumns c{};
  c.part1 = nseg == 2 ? p.seg[1].part0 : p.ldp;
  c.n0 = pad16(p.seg[0].c1 - p.seg[0].c0);
  c.n1 = pad16(p.seg[1].c1 - p.seg[1].c0);
  c.out1 = out1;
  const int total = O * p.ldp;
  grad_weight_reduce_kernel<<<(total + 31) / 32, dim3(32, kSumSlices), 0, st>>>(p.partial, (int)splits, O, p.Opad, p.ldp, c, ldo, out);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_grad_weight_workspace_bytes(int64_t O, int64_t k_total_padded, int max_ctas) {
  if (O <= 0 || k_total_padded <= 0 || max_ctas <= 0) return 256;
  const int64_t cols = k_total_padded < kGwCols ? pad16(k_total_padded) : kGwCols;
  const int64_t mtiles = (O + 127) / 128;
  return 256 + (max_ctas > 2 * mtiles ? max_ctas : 2 * mtiles) * 128 * cols * 4;
}

int exact_grad_weight_from_packed(const float* g, int64_t N, int64_t O, const uint8_t* packed0, const uint16_t* scale0,
                                  const uint16_t* min0, int64_t k0, const uint8_t* packed1, const uint16_t* scale1,
                                  const uint16_t* min1, int64_t k1, int bits, void* workspace, int64_t workspace_bytes,
                                  float* out, int64_t ldo, void* stream) {
  EXB_REQUIRE(bits == 1 || bits == 2 || bits == 4 || bits == 8, "bits must be 1, 2, 4 or 8 (got %d)", bits);
  EXB_REQUIRE(N >= 0 && O > 0 && k0 > 0 && k1 >= 0, "grad_weight_from_packed: bad shape");
  const int64_t k0pad = (k0 + 15) / 16 * 16;
  const int64_t kpad = k0pad + (k1 > 0 ? (k1 + 15) / 16 * 16 : 0);
  EXB_REQUIRE(ldo >= kpad, "grad_weight_from_packed: ldo must be at least %lld (the column blocks are padded to 16)", (long long)kpad);
  if (O % 4 != 0 || O > 256 || (reinterpret_cast<uintptr_t>(g) & 15) != 0)
    return fail(EXB_ERR_UNSUPPORTED, "grad_weight_from_packed: needs O %% 4 == 0, O <= 256 and a 16-byte aligned g (O = %lld)", (long long)O);
  if (k0 > (1 << 20) || k1 > (1 << 20))
    return fail(EXB_ERR_UNSUPPORTED, "grad_weight_from_packed: too many activation columns (k = %lld + %lld)", (long long)k0, (long long)k1);
  EXB_REQUIRE(g && packed0 && scale0 && min0 && workspace && out, "grad_weight_from_packed: null pointer");
  EXB_REQUIRE(k1 == 0 || (packed1 && scale1 && min1), "grad_weight_from_packed: null pointer in the second activation");
  EXB_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "grad_weight_from_packed: workspace must be 256-byte aligned");
  EXB_REQUIRE(N < 2147483647LL - (kGwPrefetch + 1) * kGwRows, "grad_weight_from_packed: too many rows");   // coordinates are 32-bit
  cudaStream_t st = (cudaStream_t)stream;
  GwSegment s0{}, s1{};
  s0.packed = packed0; s0.scale_bf16 = scale0; s0.min_bf16 = min0; s0.pitch = k0; s0.c1 = (int)k0;
  s1.packed = packed1; s1.scale_bf16 = scale1; s1.min_bf16 = min1; s1.pitch = k1; s1.c1 = (int)k1;
  // as many columns a launch as there are CTAs for
  const int mtiles = (int)((O + 127) / 128), cap = gw_max_cols(bits);
  int tiles = sm_count() / mtiles;
  if (tiles < 2) tiles = 2;
  if ((k0 + cap - 1) / cap + (k1 + cap - 1) / cap <= tiles)
    return gw_launch(g, N, (int)O, s0, k1 > 0 ? &s1 : nullptr, bits, workspace, workspace_bytes, out, ldo, k0pad, st);
  for (int i = 0; i < (k1 > 0 ? 2 : 1); i++) {
    const int64_t k = i ? k1 : k0;
    for (int64_t c = 0; c < k; c += (int64_t)tiles * cap) {
      GwSegment s = i ? s1 : s0;
      s.c0 = (int)c;
      s.c1 = (int)(k - c < (int64_t)tiles * cap ? k : c + (int64_t)tiles * cap);
      const int rc = gw_launch(g, N, (int)O, s, nullptr, bits, workspace, workspace_bytes, out + (i ? k0pad : 0) + c, ldo, 0, st);
      if (rc) return rc;
    }
  }
  return EXB_OK;
}

}  // extern "C"

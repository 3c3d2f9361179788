// Dense layer GEMM with fp32-equivalent accuracy on the tensor cores (three fp16 products):
//
//     C[M, N] (+)= A[M, K] B[N, K]^T  (+ A2[M, K2] B2[N, K2]^T)  (+ bias[N])
//
// Replaces the fp32 cuBLAS GEMMs of the quantised linear layer: F.linear in qlinear.forward
// (exact/exact/ops.py:150) and grad_input = grad_output.mm(weight) of linear_backward
// (exact/exact/cpp_extension/backward_func.cc:86).  M is the number of node rows (millions), K and N are
// feature widths (<= 256 per call for N).
//
// The interface, and the kernel of the contractions that are summed in chunks (k_chunk > 0); linear_tf32.cu has the other one.
//
// Arithmetic.  A row of A is scaled by a power of two per K tile (64 columns), a row of B by one for all of them, so that the
// largest element lies in [2^14, 2^15); then every operand is split into an fp16 head and an fp16 tail,
//     a = a_hi + a_lo,   a_hi = rn_f16(a),   a_lo = rn_f16(a - a_hi)      (22 bits),
// and a K tile's product is a_lo b_hi + a_hi b_lo + a_hi b_hi, accumulated in TMEM in this order: the tensor core truncates its
// fp32 accumulator, at the size of what is there already.  The K tile's sum is read back, gets its average loss (2^-23) and its
// scales back, and is added to the others in fp32 registers.  Against fp64 (Frobenius; M = 100,000 rows of the layers' operands):
// 1.04e-7 .. 1.2e-7 at 33 to 602 columns.  tf32 heads and tails in one chain, 3e-7 .. 4.4e-6; in
// chains of 64 columns, the former kernel of evaluation, 1.04e-7 .. 1.39e-7; the library's fp32 GEMM 9e-8 (48) .. 4.4e-7 (602).
// Elements that share a power of two share its range: below 2^-17 of the largest one an element has fewer than those 22 bits, and
// beside one of 2^39 times its size none.  That shows where the large ones are not in the sum: where the weight has a wide range itself
// (all tiles are then done in tf32: kind::tf32, heads and tails of 11 bits each with an exponent of their own, K tiles of 32 columns), and
// in a tile of A in which it is more than a rare element (kLinLost) while the weight has zeros or small elements to go with large ones
// (such tiles are done again in tf32, and the first way's result is not stored).  So are tiles with rows from 2^96 on, whose sums could
// overflow under B's scale.  1.1e-7 .. 1.35e-7 whatever the range.  2,449,029 x 256 -> 256: plain 1,170 us, all tiles twice
// 3,240, wide weight 2,710; 169,343 x 256 -> 256: 91, 245, 199.  (Tiles of gradients, whose magnitudes often differ that much, are
// looked through under weak weights only: done again without that rule they cost a 169,343-node GCN step 42 of 2,330 us.)
// Non-finite inputs stay non-finite and confined to their rows, but an infinite element turns its output row into NaN where an fp32
// GEMM gives +-inf (its tail is inf - inf).
//
// Structure (one CTA per SM, persistent over 128-row tiles of A, 20 warps).  Two CTAs of a cluster work as a pair on two
// neighbouring tiles (tcgen05.mma.cta_group::2, M = 256): each holds its rows of A and half of the rows of B, so a CTA fetches and
// its tensor core reads half as much of B.
//   warp 0     producer.  Shared memory is a 192 KB ring of K-tile stages; a 64-column K tile uses A (two raw fp32 boxes
//              [128 x 32] by TMA, which the heads and tails replace) and B_hi and B_lo (the CTA's rows x 64, one contiguous
//              run): three stages at Npad = 256, four for narrow outputs.  128-byte swizzle, no multicast.  The boxes of two K
//              tiles ahead are requested into L2: A is read from HBM exactly once and the ring is only a few K tiles deep.
//              Products of one K tile do without, a stage is a tile there (600,000 x 48 -> 256: 150 us, 157 with).
//   warp 1     MMA issuer (of the pair's first CTA): kind::f16, N = Npad, K = 16; 12 MMAs per K tile (with tf32, K = 8, it was as
//              many per 32 columns, and the tensor pipe was what wide products were bound by), then two commits: one frees the
//              stage (in both CTAs), one hands the accumulator over.  Accumulators are double-buffered in TMEM.
//   warps 4-11 converters: find a row's largest magnitude in the K tile (four lanes own it), scale, split, write the heads and
//              tails in place, fence.proxy.async, signal.  Two groups of four take alternate K tiles: a K tile is a chain of
//              wait, reads, conversions, stores, fence and arrival.  The first warp of a group also waits for B, so that the
//              issuing thread has one wait per K tile.  They also look for elements that fp16 cannot hold, and
//              make the tiles of B for those of A in tf32, from the weight itself.
//   warps 12-19 epilogue: add every K tile up, 128 sums a thread (registers moved to them by setmaxnreg); then the scales of the
//              columns and the bias, a staging tile per warp and a TMA store of 32 x 32 boxes: with plain stores from the
//              staging tiles the write-out was what narrow operands were bound by (2,449,029 x 48 -> 256: 904 us, boxes 589).
//              Rows whose width or pitch is no multiple of 16 bytes, and an addend, take plain stores.
// Bound by the chains of the roles: 2,250 cycles a K tile against 1,400 for its bytes (one launch of 128 columns, evaluation).
// Measured (us, tf32 -> now): 2,449,029 x 256 -> 256: 1,283 -> 1,058, with a second operand pair of 256 2,424 -> 1,826; 48 -> 256:
// 607 -> 589; 256 -> 80: 794 -> 677, 256 -> 47 (pitch 47): 683 -> 574, with an addend 1,750 -> 1,110; 232,965 x 602 -> 256: 275 -> 220
// (in chunks, evaluation: 458), 169,343 x 128 -> 256: 67 -> 63.
// Not kept: one scale per row over the whole contraction, found ahead by four more warps, and one chain in TMEM: 2,424 -> 3,561;
// sixteen epilogue warps with 64 sums a thread: 1,058 -> 1,115.
// The weight is scaled, split, padded and laid out as the tiles (both ways) once per call by a preparation kernel; the product's CTAs
// start while it runs and wait for it once they are set up (4,096 x 128 -> 64: 17.4 us one after the other, 15.4 so).
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, all roles leave their loops,
// bulk copies in flight are waited for (bounded), TMEM is freed and the status word is set.
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "exact_b200.h"
#include "tc.cuh"

namespace exb {

constexpr int kLinTileM = 128;
constexpr int kLinTileK = 64;                   // 128 bytes of halves
constexpr int kLinBoxK = 32;                    // 128 bytes of fp32: two boxes per K tile
constexpr int kLinConvGroup = 4;                // converter warps of a group; two groups take alternate K tiles
constexpr int kLinEpiGroups = 2;                // four warps each (one per 32 lanes of TMEM), alternate column blocks
// Warp groups: 0 TMA and MMA (two warps idle), 1 and 2 converters, 3 and 4 epilogue; registers move to the last, which hold the sums.
constexpr int kLinFirstConv = 4, kLinFirstEpi = 12;
constexpr int kLinThreads = (4 + 2 * kLinConvGroup + 4 * kLinEpiGroups) * 32;
constexpr int kLinRegsIssue = 32, kLinRegsConv = 64, kLinRegsEpi = 160;       // of 96 at launch: 32 + 2 x 64 + 2 x 160 = 5 x 96
static_assert(kLinRegsIssue + 2 * kLinRegsConv + 2 * kLinRegsEpi <= 5 * 96, "register split above the launch's total");
constexpr int kLinSlots = 6;                    // ring capacity in 32 KB units
constexpr int kLinMaxStages = 4;
constexpr uint32_t kLinSlotBytes = 32 * 1024;
constexpr uint32_t kLinHalf = 16 * 1024;        // of an A slot: a raw box, then the heads; the other box, then the tails
constexpr float kLinGain = 1.00000011920929f;   // 1 + 2^-23: gives back what a K tile loses to the truncating accumulator on average
constexpr int kLinPrefetch = 2;                 // K tiles of A requested into L2 ahead of their TMA load
constexpr int kLinScales = 8;                   // K tiles whose row scales are kept
constexpr int kLinHeadExp = 14;                 // the largest element of a row of a K tile is scaled to [2^14, 2^15)
// Tiles whose elements fp16 cannot hold are done again in tf32 (kind::tf32, K = 8): a K tile is 32 columns, 128 bytes as well.
constexpr int kLinWideK = 32;
constexpr int kLinWideExp = -8;                 // there the row's largest goes to [2^-8, 2^-7): no product with an fp32 number overflows
// What makes a tile of A wide: so many hits.  Of the 128 pieces of 16 columns of a row in a K tile's 32 rows: those with an element with
// lost bits, looking at half of a piece's columns, in eight rows at one and in eight rows at the other half.  (Normally
// distributed values: 0.015 hits; a column that is small beside the others: 16; a row in which most are small beside one: 4.)  Of a
// row of B: elements with lost bits.  And a row of either whose largest is 2^96 or more: sums, which carry B's scale, could overflow.
constexpr int kLinLost = 3;
constexpr int kLinFlagWords = 32;               // tiles of a CTA in a launch: one bit each

constexpr int kLinMaxCols = 256;                // of a launch

struct LinParams {
  const __half* b;         // heads and tails of the weight, as linear_prepare_kernel lays them out
  const float* col_inv;   // [Npad] what the columns were scaled by, inverted
  const int* b_range;      // [Npad] what linear_prepare_kernel says about the rows of B
  const float *B, *B2;     // the weight itself, for tiles in tf32: B[n * ldb + k * incb]
  long long ldb, incb, ldb2, incb2;
  int K, K2;
  float* C;
  const float* bias_pad;   // [Npad], with zeros behind, or null
  int* status;
  int* lib_status;    // library-wide status word of this device (capi.cu), or null
  long long M, ldc;
  int N, Npad;
  int kblocks1, kblocks;   // K tiles of the first operand pair, and of both pairs together
  int wide_kblocks1, wide_kblocks;   // the same in tf32
  int num_tiles;
  int after_prepare;       // this launch started while the preparation was running
  int bulk_out;            // C is stored by TMA: rows on 16-byte boundaries and nothing to add
  const float* addend;     // [M, ldadd] added to the product (C itself: C += ...), or null
  long long ldadd;
  int stages;              // K tiles the ring holds
  unsigned b_slot;         // bytes of a B_hi / B_lo slot: 128 per row of B in this CTA
  unsigned stage_bytes;    // A slot (32 KB) + two B slots
  unsigned tmem_cols;
};

// The exponent (biased) of the power of two that brings a largest magnitude (its bits) to [2^HEAD, 2^(HEAD + 1)), between 2^-120 and
// 2^120; of 1 for zero.  (Under an infinite one any will do: its NaN tail makes the result NaN.)
template <int HEAD>
__device__ __forceinline__ uint32_t lin_scale_exp(uint32_t magnitude) {
  const int e = (int)(magnitude >> 23);
  if (magnitude == 0) return 127u;
  const int up = e == 255 ? 120 : min(HEAD + 127 - e, 120);
  return (uint32_t)((HEAD < 7 ? max(up, -120) : up) + 127);
}
// An fp16 head and tail hold fewer than 22 bits of a scaled element other than zero when it is below 2^-3, 2^-17 of the largest one
// that shares the scale.  In this form zero is the largest number and the sign drops out.
constexpr uint32_t kLinLostBelow = 2u * 0x3e000000u - 1u;
constexpr float kLinWeakBelow = 0.5f;            // scaled: 2^-15 of a row's largest
__device__ __forceinline__ uint32_t lin_twice_minus_one(float x) { return 2u * __float_as_uint(x) - 1u; }
// Whether the largest magnitude that was brought to [2^14, 2^15) by this is 2^96 or more.
__device__ __forceinline__ bool lin_huge(uint32_t exponent) { return exponent <= 127u + kLinHeadExp - 96u; }
__device__ __forceinline__ float lin_scale(uint32_t exponent) { return __uint_as_float(exponent << 23); }
__device__ __forceinline__ float lin_inverse(uint32_t exponent) { return __uint_as_float((254u - exponent) << 23); }
// Four scaled elements -> heads and tails, two to a word, and the lesser lin_twice_minus_one of the first and the last (ODD: of the
// two between).  A non-finite element has a NaN tail (inf - inf), so its output row is NaN.
template <bool LOOK, bool ODD>
__device__ __forceinline__ uint32_t split_f16(const float (&a)[4], f32x2 scale, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
  uint32_t least[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const f32x2 x = f2_mul(f2_pack(a[2 * e], a[2 * e + 1]), scale);
    float x0, x1;
    f2_unpack(x, x0, x1);
    if (LOOK) least[e] = lin_twice_minus_one((e != 0) != ODD ? x1 : x0);
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 back = __half22float2(h);
    f2_unpack(f2_sub(x, f2_pack(back.x, back.y)), x0, x1);
    const __half2 t = __floats2half2_rn(x0, x1);
    hi[e] = *reinterpret_cast<const uint32_t*>(&h);
    lo[e] = *reinterpret_cast<const uint32_t*>(&t);
  }
  return LOOK ? min(least[0], least[1]) : 0xffffffffu;
}
__device__ __forceinline__ float lin_rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
__device__ __forceinline__ void fence_proxy_async_smem_lin() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

template <bool PAIR>
__global__ void __launch_bounds__(kLinThreads, 1)
linear_f16x3_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_a2,
                    const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ LinParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long s_full[kLinMaxStages];    // A has landed
  __shared__ __align__(8) unsigned long long s_bfull[kLinMaxStages];   // B has landed
  __shared__ __align__(8) unsigned long long s_ready[kLinMaxStages];   // A is split (in both CTAs of a pair) and B is there
  __shared__ __align__(8) unsigned long long s_empty[kLinMaxStages];
  __shared__ __align__(8) unsigned long long s_tfull[2];
  __shared__ __align__(8) unsigned long long s_tempty[2];
  __shared__ __align__(8) unsigned long long s_sfull[kLinScales];    // a K tile's row scales are there
  __shared__ uint8_t s_scale[kLinScales][kLinTileM];    // exponents: the ring leaves little room
  __shared__ __align__(8) unsigned long long s_narrow;               // all tiles have been through the first pass
  __shared__ uint32_t s_lost[kLinFlagWords + 1];   // a bit per tile of this CTA: to be done in tf32; the last word: whether there is any
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort, s_range;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // known to be uniform
  const int rank = PAIR ? (int)cluster_rank() : 0;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t stage_base = ring + kLinSlots * kLinSlotBytes;   // 4 KB of staging per epilogue warp
  volatile int* abort_flag = &s_abort;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < kLinMaxStages; s++) {
      mbar_init(smem_u32(&s_full[s]), 1);
      mbar_init(smem_u32(&s_bfull[s]), 1);
      mbar_init(smem_u32(&s_ready[s]), PAIR ? 2 * kLinConvGroup : kLinConvGroup);   // one arrival per converter warp
      mbar_init(smem_u32(&s_empty[s]), 1);
    }
    for (int b = 0; b < kLinScales; b++) {
      mbar_init(smem_u32(&s_sfull[b]), kLinConvGroup);
    }
    mbar_init(smem_u32(&s_narrow), (PAIR ? 4 : 2) * kLinConvGroup);
    for (int w = 0; w <= kLinFlagWords; w++) s_lost[w] = 0u;
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(&s_tfull[b]), 1);
      mbar_init(smem_u32(&s_tempty[b]), (PAIR ? 8 : 4) * kLinEpiGroups);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(smem_u32(&s_tmem_base), p.tmem_cols);
    else tmem_alloc(smem_u32(&s_tmem_base), p.tmem_cols);
  }
  // Nothing that the preparation wrote is read by __ldg: a read-only load could be moved up past this.
  if (p.after_prepare) asm volatile("griddepcontrol.wait;" ::: "memory");
  // What the weight's range asks for.  1: a row of B has a wide range, or one row in sixteen has elements with lost bits (a column of B
  // that is small beside others), or a row is huge: tf32 for all tiles.  2: one row in sixteen has elements below 2^-15 of its
  // largest, or zeros.  (Of uniformly or normally distributed rows of 256 elements one in 200 and one in 50.)  One warp reads it: with
  // all of them at the same few lines of L2 the kernel took 2 us longer.
  if (warp == 2) {
    int many = 0, rows = 0, weak = 0;
#pragma unroll
    for (int h = 0; h < kLinMaxCols / 32; h++) {
      const int r = 32 * h + lane < p.Npad ? __ldcg(p.b_range + 32 * h + lane) : 0;
      many = max(many, r >> 1);
      rows += r > 1;
      weak += r & 1;
    }
    const bool all = __any_sync(0xffffffffu, many >= kLinLost) || 16 * __reduce_add_sync(0xffffffffu, rows) >= p.N;
    weak = __reduce_add_sync(0xffffffffu, weak);
    if (lane == 0) s_range = (all ? 1 : 0) | (16 * weak >= p.N ? 2 : 0);
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();     // the other CTA arrives on these barriers
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  const bool wide = __any_sync(0xffffffffu, s_range & 1) != 0, weak = (s_range & 2) != 0;     // wide is known to be uniform

  // the tiles of a pair are neighbours; one past the last (an odd number of tiles) reads zeros and stores nothing
  const int first = blockIdx.x, step = gridDim.x, tiles = PAIR ? (p.num_tiles + 1) / 2 * 2 : p.num_tiles;

  // The tiles are walked twice: in fp16 (pass 0, not with a wide weight), and then those in tf32 that fp16 could not hold.  Every
  // role goes from one pass to the next when the converters of both CTAs are through the first; a pair walks a tile again for either.
  auto lost_here = [&](int i) { return (*(volatile const uint32_t*)(s_lost + (i >> 5)) >> (i & 31) & 1u) != 0; };
  auto walks = [&](int pass, int i) {
    return pass == 0 || wide || lost_here(i) || (PAIR && (smem_of_rank(smem_u32(s_lost + (i >> 5)), rank ^ 1) >> (i & 31) & 1u) != 0);
  };
  auto second_pass = [&](bool& ok) {     // whether there is one
    if (wide) return true;
    ok = PAIR ? mbar_wait_pair(smem_u32(&s_narrow), 0u, abort_flag) : mbar_wait(smem_u32(&s_narrow), 0u, abort_flag);
    if (!ok) return false;
    return *(volatile const uint32_t*)(s_lost + kLinFlagWords) != 0 ||
           (PAIR && smem_of_rank(smem_u32(s_lost + kLinFlagWords), rank ^ 1) != 0);
  };

  if (warp < kLinFirstConv) {
  set_registers<kLinRegsIssue, false>();
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      RingStage st;
      int uses = 0;   // K tiles requested so far, at most p.stages
      bool ok = true;
      for (int pass = wide ? 1 : 0; pass < 2 && ok; pass++) {
      if (pass == 1 && !second_pass(ok)) break;
      const int kblocks = pass ? p.wide_kblocks : p.kblocks, kblocks1 = pass ? p.wide_kblocks1 : p.kblocks1;
      for (int tile = first, nth = 0; tile < tiles && ok; tile += step, nth++) {
        if (!walks(pass, nth)) continue;
        for (int kb = 0; kb < kblocks; kb++, st.next(p.stages)) {
          if (!mbar_wait(smem_u32(&s_empty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t full = smem_u32(&s_full[st.s]), bfull = smem_u32(&s_bfull[st.s]);
          const uint32_t dst = ring + (uint32_t)st.s * p.stage_bytes;
          const CUtensorMap* map = kb < kblocks1 ? &tm_a : &tm_a2;
          const int x = (kb < kblocks1 ? kb : kb - kblocks1) * (pass ? kLinWideK : kLinTileK);
          mbar_arrive_expect_tx(full, pass ? kLinHalf : 2 * kLinHalf);      // a box past the row's end is zeros
          tma_load_2d(dst, map, x, tile * kLinTileM, full);
          if (pass == 0) tma_load_2d(dst + kLinHalf, map, x + kLinBoxK, tile * kLinTileM, full);
          if (uses < p.stages) uses++;
          if (pass) {
            mbar_arrive(bfull);       // the converters make these tiles of B
            continue;
          }
          mbar_arrive_expect_tx(bfull, 2 * p.b_slot);
          bulk_load(dst + kLinSlotBytes, reinterpret_cast<const char*>(p.b) + (size_t)(PAIR ? 2 * kb + rank : kb) * (2 * p.b_slot),
                    2 * p.b_slot, bfull);
          // A comes from HBM exactly once: pull the tile that will be loaded kLinPrefetch K tiles from now into L2, so that its
          // TMA load later pays L2 latency only
          int pk = kb + kLinPrefetch, pt = tile;
          if (pk >= p.kblocks) { pk -= p.kblocks; pt += step; }
          if (pt < p.num_tiles && pk < p.kblocks) {       // not with one K tile
            const CUtensorMap* pmap = pk < p.kblocks1 ? &tm_a : &tm_a2;
            const int px = (pk < p.kblocks1 ? pk : pk - p.kblocks1) * kLinTileK;
            tma_prefetch_2d(pmap, px, pt * kLinTileM);
            tma_prefetch_2d(pmap, px + kLinBoxK, pt * kLinTileM);
          }
        }
      }
      }
      // the latest round of every stage that was used: the stage before `st` and those before it
      const long long t0 = clock64();
      for (int j = 0; j < uses; j++) {
        if (--st.s < 0) {
          st.s = p.stages - 1;
          st.ph ^= 1u;
        }
        if (PAIR && ok) {
          // the pair's commits arrive in both CTAs: none may be under way when one of them exits
          ok = mbar_wait(smem_u32(&s_empty[st.s]), st.ph, abort_flag);
        }
        if (!ok) {
          // leave no bulk copy in flight (bounded)
          while (!(mbar_try_wait(smem_u32(&s_full[st.s]), st.ph) && mbar_try_wait(smem_u32(&s_bfull[st.s]), st.ph)) &&
                 clock64() - t0 < kWaitLimitCycles) {}
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The first CTA of a pair issues for both.  The whole warp walks the loop and one elected lane issues: descriptors and
    // addresses then live in uniform registers, which the instructions take; from a branch of one lane each of the twelve
    // MMAs first moved its operands there.
    if (rank == 0) {
      const bool elected = elect_one();
      constexpr int M = PAIR ? 2 * kLinTileM : kLinTileM;
      // A K tile's products, 16 halves or 8 tf32 = 32 bytes along K inside the swizzle atom at a time.  The small ones come before the
      // large ones: the accumulator truncates at its own size.
      auto products = [&](auto mma, uint32_t at) {
        const uint64_t ahi = umma_desc_sw128(at), alo = umma_desc_sw128(at + kLinHalf), bhi = umma_desc_sw128(at + kLinSlotBytes),
                       blo = umma_desc_sw128(at + kLinSlotBytes + p.b_slot);
#pragma unroll
        for (int k = 0; k < kLinTileK / 16; k++) {
          const uint64_t o = (uint64_t)(k * 2);
          mma(alo + o, bhi + o, (uint32_t)(k != 0));
          mma(ahi + o, blo + o, 1u);
        }
#pragma unroll
        for (int k = 0; k < kLinTileK / 16; k++) mma(ahi + (uint64_t)(k * 2), bhi + (uint64_t)(k * 2), 1u);
      };
      auto wait = [&](uint32_t bar, uint32_t parity) {
        const bool there = PAIR ? mbar_wait_pair(bar, parity, abort_flag) : mbar_wait(bar, parity, abort_flag);
        return __all_sync(0xffffffffu, there) != 0;
      };
      auto commit = [&](uint32_t bar) {
        if (PAIR) umma_commit_pair(bar);
        else umma_commit(bar);
      };
      RingStage st;
      int t = 0;
      bool ok = true;
      // The next stage, when it is split and B is there.
      auto ready = [&](uint32_t& at) {
        if (!wait(smem_u32(&s_ready[st.s]), st.ph)) return false;
        tc_fence_after();
        at = ring + (uint32_t)st.s * p.stage_bytes;
        return true;
      };
      for (int pass = wide ? 1 : 0; pass < 2 && ok; pass++) {
      if (pass == 1) {
        const bool second = second_pass(ok);
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!__all_sync(0xffffffffu, second)) break;
      }
      const int kblocks = pass ? p.wide_kblocks : p.kblocks;
      for (int tile = first, nth = 0; tile < tiles && ok; tile += step, nth++) {
        if (!__any_sync(0xffffffffu, walks(pass, nth))) continue;
        for (int kb = 0; kb < kblocks; kb++) {
          const int buf = t & 1;
          if (!wait(smem_u32(&s_tempty[buf]), ((uint32_t)(t >> 1) & 1u) ^ 1u)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * p.Npad);
          t++;
          uint32_t at;
          if (!ready(at)) { ok = false; break; }
          const int s0 = st.s;
          st.next(p.stages);
          if (elected) {
            if (pass == 0) {
              products([&](uint64_t a, uint64_t b, uint32_t acc) {
                if (PAIR) umma_f16_pair(d_tmem, a, b, umma_idesc_f16(M, p.Npad), acc);
                else umma_f16(d_tmem, a, b, umma_idesc_f16(M, p.Npad), acc);
              }, at);
            } else {
              products([&](uint64_t a, uint64_t b, uint32_t acc) {
                if (PAIR) umma_tf32_pair(d_tmem, a, b, umma_idesc_tf32(M, p.Npad), acc);
                else umma_tf32(d_tmem, a, b, umma_idesc_tf32(M, p.Npad), acc);
              }, at);
            }
            commit(smem_u32(&s_empty[s0]));
            commit(smem_u32(&s_tfull[buf]));
          }
          __syncwarp();
        }
      }
      }
    }
  }
  } else if (warp < kLinFirstEpi) {
    // ---------------- converter: warps 4 .. 11 ----------------
    set_registers<kLinRegsConv, false>();
    // A row of the K tile is 64 elements in two boxes; its heads replace it in the first, its tails in the second.  Four lanes
    // of a warp own a row (eight rows a pass, four passes), read all of it and write only then, so no row is overwritten early;
    // the next pass is read before the current one is written.  Which of its four groups of four columns a lane takes first
    // depends on the row: eight lanes' reads and sixteen lanes' writes then fall into different banks.
    const int group = (warp - kLinFirstConv) / kLinConvGroup, first_warp = (warp - kLinFirstConv) % kLinConvGroup == 0;
    const int r8 = lane >> 2, part = lane & 3;
    const int row0 = (warp - kLinFirstConv) % kLinConvGroup * 32;
    RingStage st;
    int turn = group, seen = 0;   // seen: K tiles so far, up to a full ring
    int n = 0;                    // K tiles so far
    bool ok = true;
    for (int pass = wide ? 1 : 0; pass < 2 && ok; pass++) {
    if (pass == 1) {
      if (!wide && lane == 0) {
        if (PAIR) mbar_arrive_pair(smem_u32(&s_narrow));
        else mbar_arrive(smem_u32(&s_narrow));
      }
      if (!second_pass(ok)) break;
    }
    const int kblocks = pass ? p.wide_kblocks : p.kblocks;
    for (int tile = first, nth = 0; tile < tiles && ok; tile += step, nth++) {
      if (!walks(pass, nth)) continue;
      for (int kb = 0; kb < kblocks; kb++, st.next(p.stages), turn ^= 1, n++) {
        const bool again = seen >= p.stages;
        if (!again) seen++;
        if (turn) continue;
        // A parity tells a round from its neighbours only, and with an odd number of stages this group meets a stage in every
        // second round.  So first see that the other group's round has been consumed; then `full` can only be one behind.
        if (again && !mbar_wait(smem_u32(&s_empty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&s_full[st.s]), st.ph, abort_flag)) { ok = false; break; }
        const uint32_t base = ring + (uint32_t)st.s * p.stage_bytes + (uint32_t)(row0 + r8) * 128u;
        int lost = 0;
        if (pass == 1) {
          // Eight elements of a row a lane, which its heads replace; the tails go to the slot's other half.
#pragma unroll
          for (int q = 0; q < 4; q++) {
            float v[2][4], m = 0.f;
#pragma unroll
            for (int j = 0; j < 2; j++) {
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[j][0]), "=f"(v[j][1]), "=f"(v[j][2]), "=f"(v[j][3])
                           : "r"(base + (uint32_t)q * 1024u + (uint32_t)(((part + 4 * j) ^ r8) << 4)) : "memory");
#pragma unroll
              for (int e = 0; e < 4; e++) m = fmaxf(m, fabsf(v[j][e]));
            }
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            const uint32_t exponent = lin_scale_exp<kLinWideExp>(__float_as_uint(m));
            const float scale = lin_scale(exponent);
            if (part == 0) s_scale[n & (kLinScales - 1)][row0 + q * 8 + r8] = (uint8_t)exponent;
#pragma unroll
            for (int j = 0; j < 2; j++) {
              float hi[4], lo[4];
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const float x = __fmul_rn(v[j][e], scale);
                hi[e] = lin_rna_tf32(x);
                lo[e] = lin_rna_tf32(__fsub_rn(x, hi[e]));
              }
              const uint32_t to = base + (uint32_t)q * 1024u + (uint32_t)(((part + 4 * j) ^ r8) << 4);
              asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(hi[0]), "f"(hi[1]), "f"(hi[2]), "f"(hi[3]) : "memory");
              asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + kLinHalf), "f"(lo[0]), "f"(lo[1]), "f"(lo[2]), "f"(lo[3]) : "memory");
            }
          }
          // This CTA's rows of B, from memory (L2): a lane is a column, or a row where columns are the contiguous direction.
          const bool second = kb >= p.wide_kblocks1;
          const float* B = second ? p.B2 : p.B;
          const long long ldb = second ? p.ldb2 : p.ldb, incb = second ? p.incb2 : p.incb;
          const int k0 = (second ? kb - p.wide_kblocks1 : kb) * kLinWideK, K = second ? p.K2 : p.K;
          const int rows = (int)(p.b_slot / 128), n0 = rank * rows, w4 = (warp - kLinFirstConv) % kLinConvGroup;
          const uint32_t bdst = ring + (uint32_t)st.s * p.stage_bytes + kLinSlotBytes;
          auto put = [&](int r, int k) {
            const float x = n0 + r < p.N && k0 + k < K ? __ldg(B + (long long)(n0 + r) * ldb + (long long)(k0 + k) * incb) : 0.f;
            const float head = lin_rna_tf32(x), tail = lin_rna_tf32(__fsub_rn(x, head));
            const uint32_t to = bdst + (uint32_t)r * 128u + (uint32_t)(((k >> 2) ^ (r & 7)) << 4) + (uint32_t)(k & 3) * 4u;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(to), "f"(head) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(to + p.b_slot), "f"(tail) : "memory");
          };
          if (incb == 1) {
#pragma unroll 4
            for (int r = w4; r < rows; r += kLinConvGroup) put(r, lane);
          } else {
            for (int r = w4 * 32 + lane; r < rows; r += kLinConvGroup * 32) {
#pragma unroll 4
              for (int k = 0; k < kLinWideK; k++) put(r, k);
            }
          }
        } else {
        float a[2][4][4];
        auto read = [&](int pass, float (&v)[4][4]) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int box = (j >> 1) ^ (r8 >> 1 & 1), c = part + 4 * ((j & 1) ^ (r8 & 1));
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[j][0]), "=f"(v[j][1]), "=f"(v[j][2]), "=f"(v[j][3])
                         : "r"(base + (uint32_t)pass * 1024u + (uint32_t)box * kLinHalf + (uint32_t)((c ^ r8) << 4)) : "memory");
          }
        };
        auto convert = [&](auto look) {
        constexpr bool LOOK = decltype(look)::value;
        read(0, a[0]);
#pragma unroll
        for (int pass = 0; pass < 4; pass++) {
          float(&v)[4][4] = a[pass & 1];
          if (pass < 3) read(pass + 1, a[(pass + 1) & 1]);
          // inf reaches the maximum, NaN does not; both stay what they are under any scale
          float m = 0.f;
#pragma unroll
          for (int j = 0; j < 4; j++) m = fmaxf(fmaxf(m, fmaxf(fabsf(v[j][0]), fabsf(v[j][1]))), fmaxf(fabsf(v[j][2]), fabsf(v[j][3])));
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));    // the four lanes of a row have read it
          const uint32_t exponent = lin_scale_exp<kLinHeadExp>(__float_as_uint(m));
          const float scale = lin_scale(exponent);
          if (part == 0) s_scale[n & (kLinScales - 1)][row0 + pass * 8 + r8] = (uint8_t)exponent;
          const f32x2 s2 = f2_pack(scale, scale);
          uint32_t least[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int box = (j >> 1) ^ (r8 >> 1 & 1), c = part + 4 * ((j & 1) ^ (r8 & 1));
            uint32_t hi[2], lo[2];
            least[j] = pass & 1 ? split_f16<LOOK, true>(v[j], s2, hi, lo) : split_f16<LOOK, false>(v[j], s2, hi, lo);
            const uint32_t to = base + (uint32_t)pass * 1024u + (uint32_t)(((box * 4 + (c >> 1)) ^ r8) << 4) + (uint32_t)(c & 1) * 8u;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to), "r"(hi[0]), "r"(hi[1]) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to + kLinHalf), "r"(lo[0]), "r"(lo[1]) : "memory");
          }
          lost += lin_huge(exponent) ? kLinLost : LOOK && min(min(least[0], least[1]), min(least[2], least[3])) < kLinLostBelow ? 1 : 0;
        }
        };
        // Elements with lost bits are looked for only under a weak weight.  Else the row's largest element meets at least 2^-15 of the
        // largest weight, and what another one lost is below 2^-24 of that product.
        if (weak) convert(std::true_type());
        else convert(std::false_type());
        }
        fence_proxy_async_smem_lin();  // generic-proxy stores -> visible to the tensor core's reads
        __syncwarp();
        if (pass == 0 && first_warp && !mbar_wait(smem_u32(&s_bfull[st.s]), st.ph, abort_flag)) { ok = false; break; }   // for the MMA's one wait
        if (lane == 0) {
          if (PAIR) mbar_arrive_leader(smem_u32(&s_ready[st.s]));
          else mbar_arrive(smem_u32(&s_ready[st.s]));
        }
        lost = __reduce_add_sync(0xffffffffu, lost);
        if (lane == 0) {
          if (lost >= kLinLost) {
            atomicOr(&s_lost[nth >> 5], 1u << (nth & 31));
            s_lost[kLinFlagWords] = 1u;
          }
          mbar_arrive(smem_u32(&s_sfull[n & (kLinScales - 1)]));
        }
      }
    }
    }
  } else {
    // ---------------- epilogue ----------------
    set_registers<kLinRegsEpi, true>();
    const int quad = warp & 3;   // TMEM lanes 32*quad .. 32*quad+31
    const int share = (warp - kLinFirstEpi) / 4;   // every kLinEpiGroups-th block of columns
    const uint32_t stage_addr = stage_base + (uint32_t)(share * 4 + quad) * 4096u;
    int t = 0;
    bool ok = true;
    // 16 columns of this thread's row to the warp's staging tile
    auto stage16 = [&](int h, const float* v) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t ci = (uint32_t)(h * 4 + j);
        const uint32_t addr = stage_addr + (uint32_t)lane * 128u + ((ci ^ ((uint32_t)lane & 7u)) << 4);
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v[4 * j]), "f"(v[4 * j + 1]),
                     "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                     : "memory");
      }
    };
    // The staged columns c0 .. c0 + cols - 1 of the warp's 32 rows, scaled (+ bias), to C: where it cannot be stored as a box, and
    // nothing is added.  A lane is a column: a store is one run of a row, whatever the row's pitch.
    auto write_out = [&](int c0, int cols, long long row_base, const float* col_inv) {
      __syncwarp();
      const int c = c0 + lane;
      const bool inside = lane < cols && c < p.N;
      const float inv = inside && col_inv != nullptr ? col_inv[c] : 1.f, bias = inside && p.bias_pad != nullptr ? p.bias_pad[c] : 0.f;
      const int rows = !inside ? 0 : p.M - row_base < 32 ? (int)(p.M - row_base) : 32;
      float* d = p.C + row_base * p.ldc + c;
#pragma unroll
      for (int r = 0; r < 32; r++, d += p.ldc) {
        float o;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(o) : "r"(stage_addr + (uint32_t)r * 128u + ((((uint32_t)lane >> 2) ^ ((uint32_t)r & 7u)) << 4) + ((uint32_t)lane & 3u) * 4u));
        if (r < rows) *d = __fmaf_rn(o, inv, bias);      // the product is exact
      }
      __syncwarp();
    };
    // The same with an addend.  A lane is a column here, and 16 rows of the addend are read before they are written (C may be the
    // addend): with four at a time 2,449,029 x 256 -> 47 took 1,440 us, 1,000 this way.
    auto add_out = [&](int c0, int cols, long long row_base, const float* col_inv) {
      __syncwarp();
      const int c = c0 + lane;
      const bool inside = lane < cols && c < p.N;
      const float inv = inside && col_inv != nullptr ? col_inv[c] : 1.f, bias = inside && p.bias_pad != nullptr ? p.bias_pad[c] : 0.f;
      const int rows = p.M - row_base < 32 ? (int)(p.M - row_base) : 32;
      float* d = p.C + row_base * p.ldc + c;
      const float* add = p.addend + row_base * p.ldadd + c;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        float old[16];
#pragma unroll
        for (int i = 0; i < 16; i++) old[i] = inside && 16 * half + i < rows ? add[(16 * half + i) * p.ldadd] : 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const int r = 16 * half + i;
          float o;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(o) : "r"(stage_addr + (uint32_t)r * 128u + ((((uint32_t)lane >> 2) ^ ((uint32_t)r & 7u)) << 4) + ((uint32_t)lane & 3u) * 4u));
          if (inside && r < rows) d[r * p.ldc] = __fmaf_rn(o, inv, bias) + old[i];
        }
      }
      __syncwarp();
    };
    auto release = [&](int buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_leader(smem_u32(&s_tempty[buf]));
        else mbar_arrive(smem_u32(&s_tempty[buf]));
      }
    };
    for (int pass = wide ? 1 : 0; pass < 2 && ok; pass++) {
    if (pass == 1 && !second_pass(ok)) break;
    const int kblocks = pass ? p.wide_kblocks : p.kblocks;
    const float* const col_inv = pass ? nullptr : p.col_inv;      // tf32: not scaled
    for (int tile = first, nth = 0; tile < tiles && ok; tile += step, nth++) {
      if (!walks(pass, nth)) continue;
      const long long row_base = (long long)tile * kLinTileM + quad * 32;
      // Every K tile is drained and added up here in fp32, with its scales and its average loss given back: half of a row's 256
      // columns a thread.  (Kept in memory the sums were 16 TB/s of L2 traffic.)
      float run[kLinMaxCols / kLinEpiGroups];
#pragma unroll
      for (int i = 0; i < kLinMaxCols / kLinEpiGroups; i++) run[i] = 0.f;
      for (int kb = 0; kb < kblocks; kb++, t++) {
        const int buf = t & 1;
        if (!mbar_wait(smem_u32(&s_tfull[buf]), (uint32_t)(t >> 1) & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        // Written well before: the scales of eight K tiles are kept, and a converter is at most four K tiles ahead of the MMAs and
        // those two of this.
        if (!mbar_wait(smem_u32(&s_sfull[t & (kLinScales - 1)]), (uint32_t)(t / kLinScales) & 1u, abort_flag)) { ok = false; break; }
        const float gain = kLinGain * lin_inverse(s_scale[t & (kLinScales - 1)][quad * 32 + lane]);
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.Npad);
#pragma unroll
        for (int q = 0; q < kLinMaxCols / kLinEpiGroups / 16; q++) {
          const int c0 = (q >> 1) * 64 + share * 32 + (q & 1) * 16;
          if (c0 < p.Npad) {
            float v[16];
            tmem_ld16(taddr + (uint32_t)c0, v);
#pragma unroll
            for (int e = 0; e < 16; e++) run[16 * q + e] = __fmaf_rn(v[e], gain, run[16 * q + e]);
          }
        }
        release(buf);
      }
      if (!ok) break;
      if ((wide || lost_here(nth)) != (pass == 1)) continue;   // the other pass stores it (all converters of the tile's rows have been here)
#pragma unroll
      for (int b = 0; b < kLinMaxCols / kLinEpiGroups / 32; b++) {
        const int c0 = b * 64 + share * 32;
        if (c0 >= p.Npad) continue;
        if (p.bulk_out) {
          // scaled here, a row per thread, and stored as a box: 128-byte rows in the staging tile's swizzle, clipped at M and N
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the box before has left the tile
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int c = c0 + 4 * j;
            float4 inv = make_float4(1.f, 1.f, 1.f, 1.f), bias = make_float4(0.f, 0.f, 0.f, 0.f);
            if (col_inv != nullptr && c < p.Npad) inv = *reinterpret_cast<const float4*>(col_inv + c);
            if (p.bias_pad != nullptr && c < p.Npad) bias = *reinterpret_cast<const float4*>(p.bias_pad + c);
            const float* v = run + 32 * b + 4 * j;
            const uint32_t addr = stage_addr + (uint32_t)lane * 128u + (((uint32_t)j ^ ((uint32_t)lane & 7u)) << 4);
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(__fmaf_rn(v[0], inv.x, bias.x)),
                         "f"(__fmaf_rn(v[1], inv.y, bias.y)), "f"(__fmaf_rn(v[2], inv.z, bias.z)), "f"(__fmaf_rn(v[3], inv.w, bias.w))
                         : "memory");
          }
          fence_proxy_async_smem_lin();
          __syncwarp();
          if (lane == 0 && row_base < p.M) tma_store_2d(&tm_c, c0, (int)row_base, stage_addr);
          if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        } else {
          stage16(0, run + 32 * b);
          stage16(1, run + 32 * b + 16);
          const int cols = p.Npad - c0 < 32 ? p.Npad - c0 : 32;
          if (p.addend != nullptr) add_out(c0, cols, row_base, col_inv);
          else write_out(c0, cols, row_base, col_inv);
        }
      }
    }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // before the staging tile goes away
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, p.tmem_cols);
    else tmem_dealloc(tmem_base, p.tmem_cols);
  }
  if (PAIR) cluster_sync();
  if (threadIdx.x == 0 && s_abort) {
    atomicExch(p.status, 1);
    raise_status(p.lib_status, EXB_STATUS_LINEAR);
  }
}

// Heads and tails of [B | B2] (rows = output features), each row scaled by a power of two, zero padded to [Npad, Kpad1 + Kpad2], in
// the order and with the swizzle of the shared-memory tiles: K tile by K tile, in it the share of each CTA of a pair (b_rows rows),
// in that the heads and then the tails, so that a CTA's part of a K tile is one contiguous run.  A block per row; also writes the
// inverse scales, what the row's range is (twice the number of elements with lost bits, kLinLost for a huge row, + 1 with an
// element that is weak), and clears the status word, if given.
constexpr int kLinPrepThreads = 128;
struct LinPrep {
  const float *B, *B2, *bias;
  long long ldb, incb, ldb2, incb2;
  int K, K2, N, Npad, Kpad1, Kpad, b_rows;
  __half* out;
  float *col_inv, *bias_pad;
  int *range, *status;
};
__global__ void __launch_bounds__(kLinPrepThreads) linear_prepare_kernel(const __grid_constant__ LinPrep p) {
  __shared__ uint32_t s_max[kLinPrepThreads / 32], s_lost[kLinPrepThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the product's CTAs set up their barriers and TMEM meanwhile
  const int n = blockIdx.x;
  if (n == 0 && threadIdx.x == 0 && p.status != nullptr) *p.status = 0;
  auto element = [&](int kk) {
    if (n >= p.N) return 0.f;
    if (kk < p.Kpad1) return kk < p.K ? __ldg(p.B + (long long)n * p.ldb + kk * p.incb) : 0.f;
    return kk - p.Kpad1 < p.K2 ? __ldg(p.B2 + (long long)n * p.ldb2 + (kk - p.Kpad1) * p.incb2) : 0.f;
  };
  uint32_t m = 0, lost = 0;
  bool weak = false;
  for (int kk = threadIdx.x; kk < p.Kpad; kk += kLinPrepThreads) m = max(m, __float_as_uint(element(kk)) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kLinPrepThreads / 32; w++) m = max(m, s_max[w]);
  const uint32_t exponent = lin_scale_exp<kLinHeadExp>(m);
  const float scale = lin_scale(exponent);
  const int share = n / p.b_rows, r = n - share * p.b_rows, shares = p.Npad / p.b_rows;
  for (int kk = threadIdx.x; kk < p.Kpad; kk += kLinPrepThreads) {
    const float x = element(kk), v = x * scale;
    lost += lin_twice_minus_one(v) < kLinLostBelow ? 1u : 0u;
    weak |= fabsf(v) < kLinWeakBelow && (kk < p.Kpad1 ? kk < p.K : kk - p.Kpad1 < p.K2);
    const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
    const int kb = kk / kLinTileK, e = kk - kb * kLinTileK;
    const size_t at = (size_t)(kb * shares + share) * 2 * p.b_rows * kLinTileK + r * kLinTileK + (((e >> 3) ^ (r & 7)) << 3) + (e & 7);
    p.out[at] = hi;
    p.out[at + (size_t)p.b_rows * kLinTileK] = lo;
  }
  lost = __reduce_add_sync(0xffffffffu, lost);
  if ((threadIdx.x & 31) == 0) s_lost[threadIdx.x >> 5] = lost;
  weak = __syncthreads_or(weak && m != 0) != 0;
  if (threadIdx.x == 0) {
    lost = lin_huge(exponent) ? kLinLost : 0;
#pragma unroll
    for (int w = 0; w < kLinPrepThreads / 32; w++) lost += s_lost[w];
    p.range[n] = (int)(2 * lost + (weak ? 1 : 0));
    p.col_inv[n] = lin_inverse(exponent);
    p.bias_pad[n] = p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
  }
}

namespace tf32 {   // linear_tf32.cu
int launch_linear(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                  int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                  int64_t ldadd, void* workspace, float* C, int64_t ldc, cudaStream_t st);
}

static inline int lin_kpad(long long K) { return (int)((K + kLinTileK - 1) / kLinTileK * kLinTileK); }
static inline int lin_wide_tiles(long long K) { return (int)((K + kLinWideK - 1) / kLinWideK); }

// One launch; the rest of its parameters is the same for all rows.
static int lin_launch_rows(const float* A, int64_t M, int64_t K, int64_t lda, const float* A2, int64_t K2, int64_t lda2, int64_t N,
                           const float* addend, int64_t ldadd, float* C, int64_t ldc, LinParams p, bool pair, bool after_prepare, cudaStream_t st) {
  CUtensorMap tm_a, tm_a2;
  int rc = make_tensor_map_2d_f32(&tm_a, A, (unsigned long long)K, (unsigned long long)M, (unsigned long long)lda * 4, kLinBoxK, kLinTileM);
  if (rc) return rc;
  if (K2 > 0) {
    rc = make_tensor_map_2d_f32(&tm_a2, A2, (unsigned long long)K2, (unsigned long long)M, (unsigned long long)lda2 * 4, kLinBoxK, kLinTileM);
    if (rc) return rc;
  } else {
    tm_a2 = tm_a;
  }
  CUtensorMap tm_c = tm_a;
  // a box ends at N only in whole 16-byte pieces
  const bool bulk_out = addend == nullptr && N % 4 == 0 && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  if (bulk_out) {
    rc = make_tensor_map_2d_f32(&tm_c, C, (unsigned long long)N, (unsigned long long)M, (unsigned long long)ldc * 4, 32, 32);
    if (rc) return rc;
  }

  p.after_prepare = after_prepare ? 1 : 0;
  p.C = C; p.M = M; p.ldc = ldc; p.addend = addend; p.ldadd = ldadd; p.bulk_out = bulk_out ? 1 : 0;
  p.num_tiles = (int)((M + kLinTileM - 1) / kLinTileM);
  const size_t dyn = (size_t)kLinSlots * kLinSlotBytes + 4 * kLinEpiGroups * 4096 + 1024;
  auto* kern = pair ? linear_f16x3_kernel<true> : linear_f16x3_kernel<false>;
  EXB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  int grid = sm_count();
  if (grid > p.num_tiles) grid = p.num_tiles;
  if (pair) grid = grid == sm_count() ? grid / 2 * 2 : (grid + 1) / 2 * 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kLinThreads);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (pair) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = 2;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    cfg.numAttrs++;
  }
  if (after_prepare) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs++;
  }
  EXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tm_a, tm_a2, tm_c, p));
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

// One preparation and its launches over checked arguments: N <= 256 columns.
static int lin_launch(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                      int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                      int64_t ldadd, void* workspace, float* C, int64_t ldc, cudaStream_t st) {
  const int Npad = (int)((N + 15) / 16 * 16);
  // Pairs need whole 16-row groups of B in each half; a single tile has no partner.
  const bool pair = M > kLinTileM && Npad % 32 == 0;
  LinPrep b{};
  b.B = B; b.B2 = B2; b.bias = bias; b.ldb = ldb; b.incb = incb; b.ldb2 = ldb2; b.incb2 = incb2;
  b.K = (int)K; b.K2 = (int)K2; b.N = (int)N; b.Npad = Npad; b.Kpad1 = lin_kpad(K); b.Kpad = b.Kpad1 + lin_kpad(K2);
  b.b_rows = pair ? Npad / 2 : Npad;   // of B in one CTA
  b.status = reinterpret_cast<int*>(workspace);
  b.col_inv = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  b.bias_pad = b.col_inv + kLinMaxCols;
  b.range = reinterpret_cast<int*>(b.bias_pad + kLinMaxCols);
  b.out = reinterpret_cast<__half*>(b.range + kLinMaxCols);
  linear_prepare_kernel<<<Npad, kLinPrepThreads, 0, st>>>(b);
  EXB_CUDA_OK(cudaGetLastError());

  LinParams p{};
  p.b = b.out; p.col_inv = b.col_inv; p.b_range = b.range; p.bias_pad = bias ? b.bias_pad : nullptr;
  p.status = b.status; p.lib_status = status_word_ptr(); p.N = (int)N; p.Npad = Npad;
  p.kblocks1 = b.Kpad1 / kLinTileK; p.kblocks = b.Kpad / kLinTileK;
  p.wide_kblocks1 = lin_wide_tiles(K); p.wide_kblocks = p.wide_kblocks1 + lin_wide_tiles(K2);
  p.B = B; p.B2 = B2; p.ldb = ldb; p.incb = incb; p.ldb2 = ldb2; p.incb2 = incb2; p.K = (int)K; p.K2 = (int)K2;
  p.b_slot = (unsigned)b.b_rows * kLinTileK * 2;
  p.stage_bytes = kLinSlotBytes + 2 * p.b_slot;
  p.stages = (int)((kLinSlots * kLinSlotBytes) / p.stage_bytes);
  if (p.stages > kLinMaxStages) p.stages = kLinMaxStages;
  unsigned cols = 32;
  while (cols < (unsigned)(2 * Npad)) cols <<= 1;
  p.tmem_cols = cols;
  // as many rows at a time as the CTAs have bits for (19.4 million on 148 SMs)
  const int64_t most = (int64_t)(sm_count() / 2 * 2) * kLinFlagWords * 32 * kLinTileM;
  for (int64_t r = 0; r < M; r += most) {
    const int rc = lin_launch_rows(A + r * lda, M - r < most ? M - r : most, K, lda, A2 ? A2 + r * lda2 : nullptr, K2, lda2, N,
                                   addend ? addend + r * ldadd : nullptr, ldadd, C + r * ldc, ldc, p, pair, r == 0, st);
    if (rc) return rc;
  }
  return EXB_OK;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_linear_workspace_bytes(int64_t N, int64_t K, int64_t K2) {
  if (N <= 0 || K <= 0 || K2 < 0) return 256;
  const int64_t Npad = (N + 15) / 16 * 16;
  // the tiles, scales and ranges of this file's kernel, and the two fp32 copies in rows of 32 columns of the other's
  const int64_t tiles = 256 + 3 * kLinMaxCols * 4 + 2 * Npad * (int64_t)(lin_kpad(K) + lin_kpad(K2)) * 2;
  const int64_t copies = 256 + 2 * Npad * (int64_t)(lin_wide_tiles(K) + lin_wide_tiles(K2)) * kLinWideK * 4;
  return tiles > copies ? tiles : copies;
}

int64_t exact_linear_partial_bytes(int64_t) { return 0; }   // the running sums of a contraction in chunks stay in registers

int exact_linear_forward(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb,
                         const float* A2, int64_t K2, int64_t lda2, const float* B2, int64_t ldb2, int64_t N,
                         const float* bias, int accumulate, void* workspace, float* C, int64_t ldc, void* stream) {
  return exact_linear_forward_strided(A, M, K, lda, B, ldb, 1, A2, K2, lda2, B2, ldb2, 1, N, bias, accumulate ? C : nullptr,
                                      accumulate ? ldc : 0, 0, nullptr, workspace, C, ldc, stream);
}

int exact_linear_forward_strided(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb,
                         const float* A2, int64_t K2, int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N,
                         const float* bias, const float* addend, int64_t ldadd, int64_t k_chunk, float* partial, void* workspace,
                         float* C, int64_t ldc, void* stream) {
  (void)partial;
  EXB_REQUIRE(k_chunk >= 0 && k_chunk % 32 == 0, "linear_forward: k_chunk must be a multiple of 32");
  EXB_REQUIRE(M >= 0 && K > 0 && N > 0 && K2 >= 0, "linear_forward: bad shape");
  if (M == 0) return EXB_OK;
  EXB_REQUIRE(A && B && C && workspace, "linear_forward: null pointer");
  EXB_REQUIRE((A2 != nullptr) == (K2 > 0) && (B2 != nullptr) == (K2 > 0), "linear_forward: the second operand pair needs A2, B2 and K2 > 0");
  EXB_REQUIRE(lda >= K && (incb != 1 || ldb >= K) && ldc >= N && (K2 == 0 || (lda2 >= K2 && (incb2 != 1 || ldb2 >= K2))), "linear_forward: leading dimension smaller than the row");
  EXB_REQUIRE(addend == nullptr || ldadd >= N, "linear_forward: leading dimension of the addend smaller than the row");
  if (N > 256) return fail(EXB_ERR_UNSUPPORTED, "linear_forward: N = %lld exceeds one MMA tile (256); call per 256-column block", (long long)N);
  if (lda % 4 != 0 || (reinterpret_cast<uintptr_t>(A) & 15) != 0 ||
      (K2 > 0 && (lda2 % 4 != 0 || (reinterpret_cast<uintptr_t>(A2) & 15) != 0)))
    return fail(EXB_ERR_UNSUPPORTED, "linear_forward: the TMA path needs 16-byte aligned rows of A (lda %% 4 == 0)");
  EXB_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "linear_forward: workspace must be 256-byte aligned");
  EXB_REQUIRE((M + kLinTileM - 1) / kLinTileM < 2147483647LL / kLinTileM, "linear_forward: too many rows");
  cudaStream_t st = (cudaStream_t)stream;
  return (k_chunk > 0 ? lin_launch : tf32::launch_linear)(A, M, K, lda, B, ldb, incb, A2, K2, lda2, B2, ldb2, incb2, N, bias, addend, ldadd,
                                                          workspace, C, ldc, st);
}

}  // extern "C"

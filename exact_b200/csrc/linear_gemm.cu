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
// chains of 64 columns, the former kernel of evaluation, 1.04e-7 .. 1.39e-7; the library's fp32 GEMM 9e-8 (48) .. 4.4e-7 (602).  The
// tail of an element is exact to 2^-39 of its row's largest one in the K tile.  Non-finite inputs stay non-finite and confined to
// their rows, but an infinite element turns its output row into NaN where an fp32 GEMM gives +-inf (its tail is inf - inf).
//
// Structure (one CTA per SM, persistent over 128-row tiles of A, 20 warps).  Two CTAs of a cluster work as a pair on two
// neighbouring tiles (tcgen05.mma.cta_group::2, M = 256): each holds its rows of A and half of the rows of B, so a CTA fetches and
// its tensor core reads half as much of B.
//   warp 0     producer.  Shared memory is a 192 KB ring of K-tile stages; a 64-column K tile uses A (two raw fp32 boxes
//              [128 x 32] by TMA, which the heads and tails replace) and B_hi and B_lo (the CTA's rows x 64, one contiguous
//              run): three stages at Npad = 256, four for narrow outputs.  128-byte swizzle, no multicast.  The boxes of two K
//              tiles ahead are requested into L2: A is read from HBM exactly once and the ring is only a few K tiles deep.
//   warp 1     MMA issuer (of the pair's first CTA): kind::f16, N = Npad, K = 16; 12 MMAs per K tile (with tf32, K = 8, it was as
//              many per 32 columns, and the tensor pipe was what wide products were bound by), then two commits: one frees the
//              stage (in both CTAs), one hands the accumulator over.  Accumulators are double-buffered in TMEM.
//   warps 4-11 converters: find a row's largest magnitude in the K tile (four lanes own it), scale, split, write the heads and
//              tails in place, fence.proxy.async, signal.  Two groups of four take alternate K tiles: a K tile is a chain of
//              wait, reads, conversions, stores, fence and arrival.  The first warp of a group also waits for B, so that the
//              issuing thread has one wait per K tile.
//   warps 12-19 epilogue: add every K tile up, 128 sums a thread (registers moved to them by setmaxnreg); then the scales of the
//              columns and the bias, a staging tile per warp and a TMA store of 32 x 32 boxes: with plain stores from the
//              staging tiles the write-out was what narrow operands were bound by (2,449,029 x 48 -> 256: 904 us, boxes 589).
//              Rows whose width or pitch is no multiple of 16 bytes, and an addend, take plain stores.
// Bound by the chains of the roles: 2,250 cycles a K tile against 1,400 for its bytes (one launch of 128 columns, evaluation).
// Measured (us, tf32 -> now): 2,449,029 x 256 -> 256: 1,283 -> 1,058, with a second operand pair of 256 2,424 -> 1,826; 48 -> 256:
// 607 -> 589; 256 -> 80: 794 -> 677, 256 -> 47 (pitch 47): 660 -> 699, with an addend 1,111 -> 1,041; 232,965 x 602 -> 256: 275 -> 220
// (in chunks, evaluation: 458), 169,343 x 128 -> 256: 67 -> 63.
// Not kept: one scale per row over the whole contraction, found ahead by four more warps, and one chain in TMEM: 2,424 -> 3,561;
// sixteen epilogue warps with 64 sums a thread: 1,058 -> 1,115.
// The weight is scaled, split, padded and laid out as the tiles once per call by a preparation kernel.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, all roles leave their loops,
// bulk copies in flight are waited for (bounded), TMEM is freed and the status word is set.
#include <cuda_fp16.h>

#include <mutex>

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

constexpr int kLinMaxCols = 256;                // of a launch

struct LinParams {
  const __half* b;         // heads and tails of the weight, as linear_prepare_kernel lays them out
  const float* col_inv;   // [Npad] what the columns were scaled by, inverted
  float* C;
  const float* bias;
  const float* bias_pad;   // [Npad], with zeros behind, or null
  int* status;
  int* lib_status;    // library-wide status word of this device (capi.cu), or null
  long long M, ldc;
  int N, Npad;
  int kblocks1, kblocks;   // K tiles of the first operand pair, and of both pairs together
  int num_tiles;
  int bulk_out;            // C is stored by TMA: rows on 16-byte boundaries and nothing to add
  const float* addend;     // [M, ldadd] added to the product (C itself: C += ...), or null
  long long ldadd;
  int stages;              // K tiles the ring holds
  unsigned b_slot;         // bytes of a B_hi / B_lo slot: 128 per row of B in this CTA
  unsigned stage_bytes;    // A slot (32 KB) + two B slots
  unsigned tmem_cols;
};

// The exponent (biased) of the power of two that brings a largest magnitude (its bits) to [2^14, 2^15); of 1 for zero and for inf
// and NaN, which stay what they are.
__device__ __forceinline__ uint32_t lin_scale_exp(uint32_t magnitude) {
  const int e = (int)(magnitude >> 23);
  if (magnitude == 0 || e == 255) return 127u;
  const int up = kLinHeadExp + 127 - e;
  return (uint32_t)((up > 120 ? 120 : up) + 127);
}
__device__ __forceinline__ float lin_scale(uint32_t exponent) { return __uint_as_float(exponent << 23); }
__device__ __forceinline__ float lin_inverse(uint32_t exponent) { return __uint_as_float((254u - exponent) << 23); }
// Four scaled elements -> heads and tails, two to a word.  A non-finite element has a NaN tail (inf - inf), so its output row is NaN.
__device__ __forceinline__ void split_f16(const float (&a)[4], f32x2 scale, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const f32x2 x = f2_mul(f2_pack(a[2 * e], a[2 * e + 1]), scale);
    float x0, x1;
    f2_unpack(x, x0, x1);
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 back = __half22float2(h);
    f2_unpack(f2_sub(x, f2_pack(back.x, back.y)), x0, x1);
    const __half2 t = __floats2half2_rn(x0, x1);
    hi[e] = *reinterpret_cast<const uint32_t*>(&h);
    lo[e] = *reinterpret_cast<const uint32_t*>(&t);
  }
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
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

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
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();     // the other CTA arrives on these barriers
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;

  // the tiles of a pair are neighbours; one past the last (an odd number of tiles) reads zeros and stores nothing
  const int first = blockIdx.x, step = gridDim.x, tiles = PAIR ? (p.num_tiles + 1) / 2 * 2 : p.num_tiles;

  if (warp < kLinFirstConv) {
  set_registers<kLinRegsIssue, false>();
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      RingStage st;
      int uses = 0;   // K tiles requested so far, at most p.stages
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        for (int kb = 0; kb < p.kblocks; kb++, st.next(p.stages)) {
          if (!mbar_wait(smem_u32(&s_empty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t full = smem_u32(&s_full[st.s]), bfull = smem_u32(&s_bfull[st.s]);
          const uint32_t dst = ring + (uint32_t)st.s * p.stage_bytes;
          mbar_arrive_expect_tx(full, 2 * kLinHalf);      // a box past the row's end is zeros
          const CUtensorMap* map = kb < p.kblocks1 ? &tm_a : &tm_a2;
          const int x = (kb < p.kblocks1 ? kb : kb - p.kblocks1) * kLinTileK;
          tma_load_2d(dst, map, x, tile * kLinTileM, full);
          tma_load_2d(dst + kLinHalf, map, x + kLinBoxK, tile * kLinTileM, full);
          mbar_arrive_expect_tx(bfull, 2 * p.b_slot);
          bulk_load(dst + kLinSlotBytes, reinterpret_cast<const char*>(p.b) + (size_t)(PAIR ? 2 * kb + rank : kb) * (2 * p.b_slot),
                    2 * p.b_slot, bfull);
          if (uses < p.stages) uses++;
          // A comes from HBM exactly once: pull the tile that will be loaded kLinPrefetch K tiles from now into L2, so that its
          // TMA load later pays L2 latency only
          int pk = kb + kLinPrefetch, pt = tile;
          if (pk >= p.kblocks) { pk -= p.kblocks; pt += step; }
          if (pt < p.num_tiles && pk < p.kblocks) {
            const CUtensorMap* pmap = pk < p.kblocks1 ? &tm_a : &tm_a2;
            const int px = (pk < p.kblocks1 ? pk : pk - p.kblocks1) * kLinTileK;
            tma_prefetch_2d(pmap, px, pt * kLinTileM);
            tma_prefetch_2d(pmap, px + kLinBoxK, pt * kLinTileM);
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
      const uint32_t idesc = umma_idesc_f16(PAIR ? 2 * kLinTileM : kLinTileM, p.Npad);
      auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
        if (PAIR) umma_f16_pair(d, a, b, idesc, acc);
        else umma_f16(d, a, b, idesc, acc);
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
      for (int tile = first; tile < tiles && ok; tile += step) {
        for (int kb = 0; kb < p.kblocks; kb++) {
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
            const uint64_t ahi = umma_desc_sw128(at), alo = umma_desc_sw128(at + kLinHalf), bhi = umma_desc_sw128(at + kLinSlotBytes),
                           blo = umma_desc_sw128(at + kLinSlotBytes + p.b_slot);
            // 16 halves = 32 bytes along K inside the swizzle atom.  The small products come before the large ones: the accumulator
            // truncates at its own size.
#pragma unroll
            for (int k = 0; k < kLinTileK / 16; k++) {
              const uint64_t o = (uint64_t)(k * 2);
              mma(d_tmem, alo + o, bhi + o, k != 0);
              mma(d_tmem, ahi + o, blo + o, 1);
            }
#pragma unroll
            for (int k = 0; k < kLinTileK / 16; k++) mma(d_tmem, ahi + (uint64_t)(k * 2), bhi + (uint64_t)(k * 2), 1);
            commit(smem_u32(&s_empty[s0]));
            commit(smem_u32(&s_tfull[buf]));
          }
          __syncwarp();
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
    for (int tile = first; tile < tiles && ok; tile += step) {
      for (int kb = 0; kb < p.kblocks; kb++, st.next(p.stages), turn ^= 1, n++) {
        const bool again = seen >= p.stages;
        if (!again) seen++;
        if (turn) continue;
        // A parity tells a round from its neighbours only, and with an odd number of stages this group meets a stage in every
        // second round.  So first see that the other group's round has been consumed; then `full` can only be one behind.
        if (again && !mbar_wait(smem_u32(&s_empty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&s_full[st.s]), st.ph, abort_flag)) { ok = false; break; }
        const uint32_t base = ring + (uint32_t)st.s * p.stage_bytes + (uint32_t)(row0 + r8) * 128u;
        float a[2][4][4];
        auto read = [&](int pass, float (&v)[4][4]) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int box = (j >> 1) ^ (r8 >> 1 & 1), c = part + 4 * ((j & 1) ^ (r8 & 1));
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[j][0]), "=f"(v[j][1]), "=f"(v[j][2]), "=f"(v[j][3])
                         : "r"(base + (uint32_t)pass * 1024u + (uint32_t)box * kLinHalf + (uint32_t)((c ^ r8) << 4)) : "memory");
          }
        };
        read(0, a[0]);
#pragma unroll
        for (int pass = 0; pass < 4; pass++) {
          float(&v)[4][4] = a[pass & 1];
          if (pass < 3) read(pass + 1, a[(pass + 1) & 1]);
          // inf reaches the maximum and leaves the row as it is; NaN does not and stays NaN under any scale
          float m = 0.f;
#pragma unroll
          for (int j = 0; j < 4; j++) m = fmaxf(fmaxf(m, fmaxf(fabsf(v[j][0]), fabsf(v[j][1]))), fmaxf(fabsf(v[j][2]), fabsf(v[j][3])));
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));    // the four lanes of a row have read it
          const uint32_t exponent = lin_scale_exp(__float_as_uint(m));
          const float scale = lin_scale(exponent);
          if (part == 0) s_scale[n & (kLinScales - 1)][row0 + pass * 8 + r8] = (uint8_t)exponent;
          const f32x2 s2 = f2_pack(scale, scale);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int box = (j >> 1) ^ (r8 >> 1 & 1), c = part + 4 * ((j & 1) ^ (r8 & 1));
            uint32_t hi[2], lo[2];
            split_f16(v[j], s2, hi, lo);
            const uint32_t to = base + (uint32_t)pass * 1024u + (uint32_t)(((box * 4 + (c >> 1)) ^ r8) << 4) + (uint32_t)(c & 1) * 8u;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to), "r"(hi[0]), "r"(hi[1]) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to + kLinHalf), "r"(lo[0]), "r"(lo[1]) : "memory");
          }
        }
        fence_proxy_async_smem_lin();  // generic-proxy stores -> visible to the tensor core's reads
        __syncwarp();
        if (first_warp && !mbar_wait(smem_u32(&s_bfull[st.s]), st.ph, abort_flag)) { ok = false; break; }   // for the MMA's one wait
        if (lane == 0) {
          mbar_arrive(smem_u32(&s_sfull[n & (kLinScales - 1)]));
          if (PAIR) mbar_arrive_leader(smem_u32(&s_ready[st.s]));
          else mbar_arrive(smem_u32(&s_ready[st.s]));
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
    // nothing is added.  Four rows at a time, four columns a lane.
    auto write_out = [&](int c0, int cols, long long row_base) {
      __syncwarp();
      const uint32_t ci = (uint32_t)lane & 7u;
      const int c = c0 + (int)ci * 4;
      const bool inside = (int)ci * 4 < cols && c < p.N;
      const float4 inv = inside ? __ldg(reinterpret_cast<const float4*>(p.col_inv + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 bias = inside && p.bias_pad != nullptr ? __ldg(reinterpret_cast<const float4*>(p.bias_pad + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int rr = 4 * i + (lane >> 3);
        float4 o;
        const uint32_t addr = stage_addr + (uint32_t)rr * 128u + ((ci ^ ((uint32_t)rr & 7u)) << 4);
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(addr));
        if (row_base + rr < p.M && inside) {
          float* d = p.C + (row_base + rr) * p.ldc + c;
          const float v[4] = {__fmaf_rn(o.x, inv.x, bias.x), __fmaf_rn(o.y, inv.y, bias.y), __fmaf_rn(o.z, inv.z, bias.z),
                              __fmaf_rn(o.w, inv.w, bias.w)};   // the products are exact
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (c + e < p.N) d[e] = v[e];
        }
      }
      __syncwarp();
    };
    // The same with an addend.  A lane is a column here, and 16 rows of the addend are read before they are written (C may be the
    // addend): with four at a time 2,449,029 x 256 -> 47 took 1,440 us, 1,000 this way.
    auto add_out = [&](int c0, int cols, long long row_base) {
      __syncwarp();
      const int c = c0 + lane;
      const bool inside = lane < cols && c < p.N;
      const float inv = inside ? __ldg(p.col_inv + c) : 0.f, bias = inside && p.bias_pad != nullptr ? __ldg(p.bias_pad + c) : 0.f;
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
    for (int tile = first; tile < tiles && ok; tile += step) {
      const long long row_base = (long long)tile * kLinTileM + quad * 32;
      // Every K tile is drained and added up here in fp32, with its scales and its average loss given back: half of a row's 256
      // columns a thread.  (Kept in memory the sums were 16 TB/s of L2 traffic.)
      float run[kLinMaxCols / kLinEpiGroups];
#pragma unroll
      for (int i = 0; i < kLinMaxCols / kLinEpiGroups; i++) run[i] = 0.f;
      for (int kb = 0; kb < p.kblocks; kb++, t++) {
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
            float4 inv = make_float4(0.f, 0.f, 0.f, 0.f), bias = inv;
            if (c < p.Npad) inv = __ldg(reinterpret_cast<const float4*>(p.col_inv + c));
            if (p.bias_pad != nullptr && c < p.Npad) bias = __ldg(reinterpret_cast<const float4*>(p.bias_pad + c));
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
          if (p.addend != nullptr) add_out(c0, cols, row_base);
          else write_out(c0, cols, row_base);
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
// inverse scales and clears the status word, if given.
constexpr int kLinPrepThreads = 128;
__global__ void __launch_bounds__(kLinPrepThreads) linear_prepare_kernel(
    const float* __restrict__ B, int K, long long ldb, long long incb, const float* __restrict__ B2, int K2, long long ldb2,
    long long incb2, int N, int Npad, int Kpad1, int Kpad, int b_rows, __half* __restrict__ out, float* __restrict__ col_inv,
    const float* __restrict__ bias, float* __restrict__ bias_pad, int* status) {
  __shared__ uint32_t s_max[kLinPrepThreads / 32];
  const int n = blockIdx.x;
  if (n == 0 && threadIdx.x == 0 && status != nullptr) *status = 0;
  auto element = [&](int kk) {
    if (n >= N) return 0.f;
    if (kk < Kpad1) return kk < K ? __ldg(B + (long long)n * ldb + kk * incb) : 0.f;
    return kk - Kpad1 < K2 ? __ldg(B2 + (long long)n * ldb2 + (kk - Kpad1) * incb2) : 0.f;
  };
  uint32_t m = 0;
  for (int kk = threadIdx.x; kk < Kpad; kk += kLinPrepThreads) m = max(m, __float_as_uint(element(kk)) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kLinPrepThreads / 32; w++) m = max(m, s_max[w]);
  const float scale = lin_scale(lin_scale_exp(m));
  if (threadIdx.x == 0) {
    col_inv[n] = lin_inverse(lin_scale_exp(m));
    bias_pad[n] = bias != nullptr && n < N ? bias[n] : 0.f;
  }
  const int share = n / b_rows, r = n - share * b_rows;
  for (int kk = threadIdx.x; kk < Kpad; kk += kLinPrepThreads) {
    const float v = element(kk) * scale;
    const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
    const int kb = kk / kLinTileK, e = kk - kb * kLinTileK;
    const size_t at = (size_t)(kb * (Npad / b_rows) + share) * 2 * b_rows * kLinTileK + r * kLinTileK + (((e >> 3) ^ (r & 7)) << 3) + (e & 7);
    out[at] = hi;
    out[at + (size_t)b_rows * kLinTileK] = lo;
  }
}

namespace tf32 {   // linear_tf32.cu
int launch_linear(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                  int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                  int64_t ldadd, void* workspace, float* C, int64_t ldc, cudaStream_t st);
}

static inline int lin_kpad(long long K) { return (int)((K + kLinTileK - 1) / kLinTileK * kLinTileK); }

// One launch over checked arguments: N <= 256 columns.
static int lin_launch(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                      int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                      int64_t ldadd, void* workspace, float* C, int64_t ldc, cudaStream_t st) {
  const int Npad = (int)((N + 15) / 16 * 16);
  const int Kpad1 = lin_kpad(K), Kpad2 = lin_kpad(K2), Kpad = Kpad1 + Kpad2;
  int* status = reinterpret_cast<int*>(workspace);
  float* col_inv = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  float* bias_pad = col_inv + kLinMaxCols;
  __half* b = reinterpret_cast<__half*>(bias_pad + kLinMaxCols);
  const int num_tiles = (int)((M + kLinTileM - 1) / kLinTileM);
  // Pairs need whole 16-row groups of B in each half; a single tile has no partner.
  const bool pair = num_tiles >= 2 && Npad % 32 == 0;
  const int b_rows = pair ? Npad / 2 : Npad;   // of B in one CTA

  linear_prepare_kernel<<<Npad, kLinPrepThreads, 0, st>>>(B, (int)K, ldb, incb, B2, (int)K2, ldb2, incb2, (int)N, Npad, Kpad1, Kpad,
                                                          b_rows, b, col_inv, bias, bias_pad, status);
  EXB_CUDA_OK(cudaGetLastError());

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

  LinParams p{};
  p.b = b; p.C = C; p.bias = bias; p.status = status; p.lib_status = status_word_ptr(); p.M = M; p.ldc = ldc; p.N = (int)N; p.Npad = Npad;
  p.kblocks1 = Kpad1 / kLinTileK; p.kblocks = Kpad / kLinTileK;
  p.num_tiles = num_tiles;
  p.addend = addend; p.ldadd = ldadd;
  p.col_inv = col_inv; p.bias_pad = bias ? bias_pad : nullptr; p.bulk_out = bulk_out ? 1 : 0;
  p.b_slot = (unsigned)b_rows * kLinTileK * 2;
  p.stage_bytes = kLinSlotBytes + 2 * p.b_slot;
  p.stages = (int)((kLinSlots * kLinSlotBytes) / p.stage_bytes);
  if (p.stages > kLinMaxStages) p.stages = kLinMaxStages;
  unsigned cols = 32;
  while (cols < (unsigned)(2 * Npad)) cols <<= 1;
  p.tmem_cols = cols;
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
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pair ? 1 : 0;
  EXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tm_a, tm_a2, tm_c, p));
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_linear_workspace_bytes(int64_t N, int64_t K, int64_t K2) {
  if (N <= 0 || K <= 0 || K2 < 0) return 256;
  const int64_t Npad = (N + 15) / 16 * 16;
  // the tiles and scales of this file's kernel, and the two fp32 copies in rows of 32 columns of the other's
  const int64_t tiles = 256 + 2 * kLinMaxCols * 4 + 2 * Npad * (int64_t)(lin_kpad(K) + lin_kpad(K2)) * 2;
  const int64_t copies = 256 + 2 * Npad * ((K + 31) / 32 * 32 + (K2 + 31) / 32 * 32) * 4;
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

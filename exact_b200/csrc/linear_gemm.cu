// Dense layer GEMM with fp32-equivalent accuracy on the tensor cores ("3xTF32"):
//
//     C[M, N] (+)= A[M, K] B[N, K]^T  (+ A2[M, K2] B2[N, K2]^T)  (+ bias[N])
//
// Replaces the fp32 cuBLAS GEMMs of the quantised linear layer: F.linear in qlinear.forward
// (exact/exact/ops.py:150) and grad_input = grad_output.mm(weight) of linear_backward
// (exact/exact/cpp_extension/backward_func.cc:86).  M is the number of node rows (millions), K and N are
// feature widths (<= 256 per call for N).
//
// Arithmetic.  Every fp32 operand is split into a tf32 head and a tf32 tail,
//     a = a_hi + a_lo,   a_hi = rna_tf32(a),   a_lo = rna_tf32(a - a_hi)      (|a_lo| <= 2^-11 |a|),
// and the product is accumulated in fp32 as  a_hi b_hi + a_lo b_hi + a_hi b_lo.  The dropped terms
// (a_lo b_lo and the rounding of the tails) are below 2^-21 |a b|, the size of the fp32 rounding of a
// plain fp32 dot product, so the result is as accurate as an fp32 SIMT GEMM at three tensor-core MMAs
// per tile instead of one fp32 FMA per product.  Non-finite inputs stay non-finite and confined to their
// rows, but an infinite element turns its output row into NaN where an fp32 GEMM gives +-inf (its tail is
// inf - inf).
//
// Structure (one CTA per SM, persistent over 128-row tiles of A, 18 warps).  Two CTAs of a cluster work as a pair on two
// neighbouring tiles (tcgen05.mma.cta_group::2, M = 256): each holds its rows of A and half of the rows of B, so a CTA fetches and
// its tensor core reads half as much of B, which is what the product is bound by once the roles keep up (at 256 x 256 the
// shared-memory traffic of a K tile takes as long as its MMAs), and the ring holds three K tiles instead of two.
//   warp 0     producer.  Shared memory is a 192 KB ring of K-tile stages; a 32-column K tile uses three
//              parts: A (raw fp32 [128 x 32] by TMA, 16 KB, the tail tile goes into the part's other half),
//              B_hi and B_lo (the CTA's rows x 32, one contiguous run): three stages at Npad = 256, four for narrow
//              outputs.  128-byte swizzle, no multicast.
//              The A tile of four K tiles ahead is requested into L2 (tensor prefetch): A is read from
//              HBM exactly once and the ring is only a few K tiles deep.
//   warps 2-9  converters: rewrite the raw A tile in place as a_hi and write a_lo beside it (same swizzled
//              offsets), fence.proxy.async, signal.  Two groups of four take alternate K tiles: a K tile is a chain of wait,
//              reads, conversions, stores, fence and arrival, 1,250 cycles whatever the width of the output.  The first
//              warp of a group also waits for B, so that the issuing thread has one wait per K tile.
//   warp 1     MMA issuer (of the pair's first CTA): kind::tf32, N = Npad, K = 8; per K tile 12 MMAs (hi*hi, lo*hi, hi*lo),
//              then one commit that frees the stage (in both CTAs).  Its chain of waits and index arithmetic was what the
//              kernel was bound by (2,500 cycles per K tile at any width; the MMAs take 1,536 at 256 columns): stage and
//              parity are counted instead of divided out.  Accumulators are double-buffered in TMEM.
//   warps 10-17 epilogue: tcgen05.ld -> per-warp staging tile in shared memory -> (+ bias, + addend)
//              -> coalesced global stores; two groups of four take alternate blocks of 32 columns.
// Measured (us, single CTAs -> now; ranges over boxes and runs): 2,449,029 x 256 -> 256: 1,673 -> 1,335 - 1,365, with a second operand
// pair of 256 3,365 -> 2,400 - 2,890; 48 -> 256: 1,046 -> 810 - 950; 256 -> 47: 1,305 -> 760 - 860; 232,965 x 604 -> 256: 368 ->
// 298 - 321; 169,343 x 128 -> 256: 100 -> 71 - 83.  With the pair alone and the chains as they were it lost (1,710 -> 2,008).
// The weight is split, padded and laid out as the tiles once per call by a preparation kernel.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, all roles leave their loops,
// bulk copies in flight are waited for (bounded), TMEM is freed and the status word is set.
#include <mutex>

#include "exact_b200.h"
#include "tc.cuh"

namespace exb {

constexpr int kLinTileM = 128;
constexpr int kLinTileK = 32;
constexpr int kLinConvWarps = 8;                // in two groups that take alternate K tiles
constexpr int kLinConvGroup = kLinConvWarps / 2;
constexpr int kLinEpiGroups = 2;                // four warps each (one per 32 lanes of TMEM), alternate column blocks
constexpr int kLinThreads = (2 + kLinConvWarps + 4 * kLinEpiGroups) * 32;   // TMA, MMA, converters, epilogue
constexpr int kLinSlots = 6;                    // ring capacity in 32 KB units
constexpr int kLinMaxStages = 4;
constexpr uint32_t kLinSlotBytes = 32 * 1024;
constexpr uint32_t kLinHalf = 16 * 1024;        // raw / tail halves of an A slot
constexpr int kLinSleepNs = 200;                // back-off between polls of the epilogue, which waits long
constexpr float kLinGain = 1.00000011920929f;   // 1 + 2^-23: gives back what a chunk of two K tiles loses to the truncating accumulator on average
constexpr int kLinChunkedCols = 128;             // columns of a launch in chunks
constexpr int kLinPrefetch = 4;                 // K tiles of A requested into L2 ahead of their TMA load

struct LinParams {
  const float* b;         // heads and tails of the weight, as linear_prepare_kernel lays them out
  float* C;
  const float* bias;
  int* status;
  int* lib_status;    // library-wide status word of this device (capi.cu), or null
  long long M, ldc;
  int N, Npad;
  int kblocks1, kblocks;   // K tiles of the first operand pair, and of both pairs together
  int num_tiles;
  const float* addend;     // [M, ldadd] added to the product (C itself: C += ...), or null
  long long ldadd;
  int chunk;               // K tiles that are accumulated in TMEM before their sum is taken over in fp32
  int stages;              // K tiles the ring holds
  unsigned b_slot;         // bytes of a B_hi / B_lo slot: 128 per row of B in this CTA
  unsigned stage_bytes;    // A slot (32 KB) + two B slots
  unsigned tmem_cols;
};

__device__ __forceinline__ uint32_t rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
// (head, tail) of the split.  A non-finite element has a NaN tail (inf - inf), so its output row is NaN.
__device__ __forceinline__ void split_tf32(float a, float& hi, float& lo) {
  hi = __uint_as_float(rna_tf32(a));
  lo = __uint_as_float(rna_tf32(__fsub_rn(a, hi)));
}
__device__ __forceinline__ void fence_proxy_async_smem_lin() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// CHUNKED: the contraction is drained from TMEM every p.chunk K tiles, in fp32 and with a chunk's average loss given back; the small
// products of two K tiles come before the large ones, as each step truncates at the size of what is there already.  With chunks of
// two K tiles 1.4e-7 and 1.3e-7 from fp64 at 602 and at 256 columns (the interleaved order and no correction: 5.2e-7, in one piece 4.4e-6 and
// 1.8e-6).  (A kernel of its own: its epilogue's
// registers and code cost the unchunked product 5 %.)
template <bool CHUNKED, bool PAIR>
__global__ void __launch_bounds__(kLinThreads, 1)
linear_tf32x3_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_a2,
                     const __grid_constant__ LinParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long s_full[kLinMaxStages];    // A has landed
  __shared__ __align__(8) unsigned long long s_bfull[kLinMaxStages];   // B has landed
  __shared__ __align__(8) unsigned long long s_ready[kLinMaxStages];   // A is split (in both CTAs of a pair) and B is there
  __shared__ __align__(8) unsigned long long s_empty[kLinMaxStages];
  __shared__ __align__(8) unsigned long long s_tfull[2];
  __shared__ __align__(8) unsigned long long s_tempty[2];
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
          mbar_arrive_expect_tx(full, kLinHalf);
          if (kb < p.kblocks1) tma_load_2d(dst, &tm_a, kb * kLinTileK, tile * kLinTileM, full);
          else tma_load_2d(dst, &tm_a2, (kb - p.kblocks1) * kLinTileK, tile * kLinTileM, full);
          mbar_arrive_expect_tx(bfull, 2 * p.b_slot);
          bulk_load(dst + kLinSlotBytes, reinterpret_cast<const char*>(p.b) + (size_t)(PAIR ? 2 * kb + rank : kb) * (2 * p.b_slot),
                    2 * p.b_slot, bfull);
          if (uses < p.stages) uses++;
          // A comes from HBM exactly once: pull the tile that will be loaded kLinPrefetch K tiles from
          // now into L2, so that its TMA load later pays L2 latency only (the ring holds three or four K tiles)
          int pk = kb + kLinPrefetch, pt = tile;
          if (pk >= p.kblocks) { pk -= p.kblocks; pt += step; }
          if (pt < p.num_tiles && pk < p.kblocks) {
            if (pk < p.kblocks1) tma_prefetch_2d(&tm_a, pk * kLinTileK, pt * kLinTileM);
            else tma_prefetch_2d(&tm_a2, (pk - p.kblocks1) * kLinTileK, pt * kLinTileM);
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
      const uint32_t idesc = umma_idesc_tf32(PAIR ? 2 * kLinTileM : kLinTileM, p.Npad);
      auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
        if (PAIR) umma_tf32_pair(d, a, b, idesc, acc);
        else umma_tf32(d, a, b, idesc, acc);
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
      auto small_products = [&](uint32_t d, uint32_t at, bool first) {
        const uint64_t ahi = umma_desc_sw128(at), alo = umma_desc_sw128(at + kLinHalf), bhi = umma_desc_sw128(at + kLinSlotBytes),
                       blo = umma_desc_sw128(at + kLinSlotBytes + p.b_slot);
#pragma unroll
        for (int k4 = 0; k4 < kLinTileK / 8; k4++) {
          const uint64_t o = (uint64_t)(k4 * 2);   // 8 tf32 = 32 bytes along K inside the swizzle atom
          mma(d, alo + o, bhi + o, !first || k4 != 0);
          mma(d, ahi + o, blo + o, 1);
        }
      };
      auto head_products = [&](uint32_t d, uint32_t at) {
        const uint64_t ahi = umma_desc_sw128(at), bhi = umma_desc_sw128(at + kLinSlotBytes);
#pragma unroll
        for (int k4 = 0; k4 < kLinTileK / 8; k4++) mma(d, ahi + (uint64_t)(k4 * 2), bhi + (uint64_t)(k4 * 2), 1);
      };
      // The next stage, when it is split and B is there.
      auto ready = [&](uint32_t& at) {
        if (!wait(smem_u32(&s_ready[st.s]), st.ph)) return false;
        tc_fence_after();
        at = ring + (uint32_t)st.s * p.stage_bytes;
        return true;
      };
      for (int tile = first; tile < tiles && ok; tile += step) {
        int buf = 0;
        uint32_t d_tmem = 0;
        for (int kb = 0; kb < p.kblocks;) {
          const bool opens = CHUNKED ? kb % p.chunk == 0 : kb == 0;
          if (opens) {
            buf = t & 1;
            const uint32_t tph = (uint32_t)(t >> 1) & 1u;
            if (!wait(smem_u32(&s_tempty[buf]), tph ^ 1u)) { ok = false; break; }
            tc_fence_after();
            d_tmem = tmem_base + (uint32_t)(buf * p.Npad);
            t++;
          }
          uint32_t at0, at1 = 0;
          if (!ready(at0)) { ok = false; break; }
          const int s0 = st.s;
          st.next(p.stages);
          if (!CHUNKED) {
            if (elected) {
              const uint64_t ahi = umma_desc_sw128(at0), alo = umma_desc_sw128(at0 + kLinHalf), bhi = umma_desc_sw128(at0 + kLinSlotBytes),
                             blo = umma_desc_sw128(at0 + kLinSlotBytes + p.b_slot);
#pragma unroll
              for (int k4 = 0; k4 < kLinTileK / 8; k4++) {
                const uint64_t o = (uint64_t)(k4 * 2);
                mma(d_tmem, alo + o, bhi + o, !opens || k4 != 0);
                mma(d_tmem, ahi + o, bhi + o, 1);
              }
#pragma unroll
              for (int k4 = 0; k4 < kLinTileK / 8; k4++) mma(d_tmem, ahi + (uint64_t)(k4 * 2), blo + (uint64_t)(k4 * 2), 1);
              commit(smem_u32(&s_empty[s0]));
              if (kb + 1 == p.kblocks) commit(smem_u32(&s_tfull[buf]));
            }
            kb++;
          } else {
            // the small products of two K tiles before the large ones: the accumulator truncates at its own size
            if (elected) small_products(d_tmem, at0, opens);
            const bool two = kb + 1 < p.kblocks && (kb + 1) % p.chunk != 0;
            const int s1 = st.s;
            if (two) {
              if (!ready(at1)) { ok = false; break; }
              st.next(p.stages);
            }
            if (elected) {
              if (two) small_products(d_tmem, at1, false);
              head_products(d_tmem, at0);
              commit(smem_u32(&s_empty[s0]));
              if (two) {
                head_products(d_tmem, at1);
                commit(smem_u32(&s_empty[s1]));
              }
            }
            kb += two ? 2 : 1;
            if (elected && (kb % p.chunk == 0 || kb == p.kblocks)) commit(smem_u32(&s_tfull[buf]));
          }
          __syncwarp();
        }
      }
    }
  } else if (warp < 2 + kLinConvWarps) {
    // ---------------- converter: warps 2 .. 2 + kLinConvWarps - 1 ----------------
    const int group = (warp - 2) / kLinConvGroup, ct = threadIdx.x - 64 - group * 32 * kLinConvGroup;
    constexpr int kPer = (int)(kLinHalf / 16) / (32 * kLinConvGroup);   // 16-byte chunks per thread
    constexpr int kBatch = 4;
    RingStage st;
    int turn = group, seen = 0;   // seen: K tiles so far, up to a full ring
    bool ok = true;
    for (int tile = first; tile < tiles && ok; tile += step) {
      for (int kb = 0; kb < p.kblocks; kb++, st.next(p.stages), turn ^= 1) {
        const bool again = seen >= p.stages;
        if (!again) seen++;
        if (turn) continue;
        // A parity tells a round from its neighbours only, and with an odd number of stages this group meets a stage in every
        // second round.  So first see that the other group's round has been consumed; then `full` can only be one behind.
        if (again && !mbar_wait(smem_u32(&s_empty[st.s]), st.ph ^ 1u, abort_flag)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&s_full[st.s]), st.ph, abort_flag)) { ok = false; break; }
        const uint32_t base = ring + (uint32_t)st.s * p.stage_bytes + (uint32_t)ct * 16u;
#pragma unroll
        for (int i0 = 0; i0 < kPer; i0 += kBatch) {
          float a[kBatch][4];
#pragma unroll
          for (int i = 0; i < kBatch; i++)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a[i][0]), "=f"(a[i][1]), "=f"(a[i][2]), "=f"(a[i][3])
                         : "r"(base + (uint32_t)(i0 + i) * (32u * kLinConvGroup * 16u)));
#pragma unroll
          for (int i = 0; i < kBatch; i++) {
            const uint32_t addr = base + (uint32_t)(i0 + i) * (32u * kLinConvGroup * 16u);
            float h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; e++) h[e] = __uint_as_float(rna_tf32(a[i][e]));
#pragma unroll
            for (int e = 0; e < 4; e += 2) {   // tails: paired subtract, then round to tf32
              float d0, d1;
              f2_unpack(f2_sub(f2_pack(a[i][e], a[i][e + 1]), f2_pack(h[e], h[e + 1])), d0, d1);
              l[e] = __uint_as_float(rna_tf32(d0));
              l[e + 1] = __uint_as_float(rna_tf32(d1));
            }
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(h[0]), "f"(h[1]), "f"(h[2]), "f"(h[3]) : "memory");
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr + kLinHalf), "f"(l[0]), "f"(l[1]), "f"(l[2]), "f"(l[3]) : "memory");
          }
        }
        fence_proxy_async_smem_lin();  // generic-proxy stores -> visible to the tensor core's reads
        __syncwarp();
        if (ct < 32 && !mbar_wait(smem_u32(&s_bfull[st.s]), st.ph, abort_flag)) { ok = false; break; }   // for the MMA's one wait
        if (lane == 0) {
          if (PAIR) mbar_arrive_leader(smem_u32(&s_ready[st.s]));
          else mbar_arrive(smem_u32(&s_ready[st.s]));
        }
      }
    }
  } else {
    // ---------------- epilogue: the last warps ----------------
    const int quad = warp & 3;   // TMEM lanes 32*quad .. 32*quad+31
    const int share = (warp - 2 - kLinConvWarps) / 4;   // every kLinEpiGroups-th block of columns
    const bool vec = (p.N & 3) == 0 && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 &&
                     (p.addend == nullptr || ((p.ldadd & 3) == 0 && (reinterpret_cast<uintptr_t>(p.addend) & 15) == 0));
    const uint32_t stage_addr = stage_base + (uint32_t)(share * 4 + quad) * 4096u;
    int t = 0;
    bool ok = true;
    const int chunks = CHUNKED ? (p.kblocks + p.chunk - 1) / p.chunk : 1;
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
    // the staged columns c0 .. c0 + cols - 1 of the warp's 32 rows (+ bias, + addend) to C
    auto write_out = [&](int c0, int cols, long long row_base) {
      __syncwarp();
      const uint32_t ci = (uint32_t)lane & 7u;
      const int c = c0 + (int)ci * 4;
      float bv[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.bias != nullptr) {
#pragma unroll
        for (int bb = 0; bb < 4; bb++)
          if (c + bb < p.N) bv[bb] = __ldg(p.bias + c + bb);
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int rr = 4 * i + (lane >> 3);
        const long long nn = row_base + rr;
        float4 o;
        const uint32_t addr = stage_addr + (uint32_t)rr * 128u + ((ci ^ ((uint32_t)rr & 7u)) << 4);
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(addr));
        if (nn < p.M && (int)ci * 4 < cols && c < p.N) {
          float* d = p.C + nn * p.ldc + c;
          const float* add = p.addend ? p.addend + nn * p.ldadd + c : nullptr;
          o.x += bv[0]; o.y += bv[1]; o.z += bv[2]; o.w += bv[3];
          if (vec) {   // N % 4 == 0, so c + 4 <= N
            if (add) {
              const float4 old = *reinterpret_cast<const float4*>(add);
              o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
            }
            __stcs(reinterpret_cast<float4*>(d), o);
          } else {
            const float ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int bb = 0; bb < 4; bb++)
              if (c + bb < p.N) d[bb] = add ? add[bb] + ov[bb] : ov[bb];
          }
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
      if constexpr (CHUNKED) {
        // At most 128 columns, so that this thread's half of a row's sums stays in registers: kept in memory they were 16 TB/s of
        // L2 traffic.  232,965 x 602 -> 256, two launches, chunks of 64: 576 -> 457 us; x 512 453 -> 377 (library: 1,235, 1,049).
        static_assert(kLinEpiGroups == 2 && kLinChunkedCols == 128, "64 columns a thread");
        float run[64];
#pragma unroll
        for (int i = 0; i < 64; i++) run[i] = 0.f;
        for (int ch = 0; ch < chunks; ch++, t++) {
          const int buf = t & 1;
          if (!mbar_wait<kLinSleepNs>(smem_u32(&s_tfull[buf]), (uint32_t)(t >> 1) & 1u, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.Npad);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int c0 = (q >> 1) * 64 + share * 32 + (q & 1) * 16;
            if (c0 < p.Npad) {
              float v[16];
              tmem_ld16(taddr + (uint32_t)c0, v);
#pragma unroll
              for (int e = 0; e < 16; e++) run[16 * q + e] = __fmaf_rn(v[e], kLinGain, run[16 * q + e]);
            }
          }
          release(buf);
        }
        if (!ok) break;
#pragma unroll
        for (int b = 0; b < 2; b++) {
          const int c0 = b * 64 + share * 32;
          if (c0 < p.Npad) {
            stage16(0, run + 32 * b);
            stage16(1, run + 32 * b + 16);
            write_out(c0, p.Npad - c0 < 32 ? p.Npad - c0 : 32, row_base);
          }
        }
      } else {
        const int buf = t & 1;
        const uint32_t ph = (uint32_t)(t >> 1) & 1u;
        t++;
        if (!mbar_wait<kLinSleepNs>(smem_u32(&s_tfull[buf]), ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.Npad);
        for (int c0 = share * 32; c0 < p.Npad; c0 += 32 * kLinEpiGroups) {
          const int cols = (p.Npad - c0) < 32 ? (p.Npad - c0) : 32;   // 16 or 32
          for (int h = 0; h * 16 < cols; h++) {
            float v[16];
            tmem_ld16(taddr + (uint32_t)(c0 + h * 16), v);
            stage16(h, v);
          }
          write_out(c0, cols, row_base);
        }
        release(buf);
      }
    }
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

// Heads and tails of [B | B2] (rows = output features), zero padded to [Npad, Kpad1 + Kpad2], in the order and with the swizzle
// of the shared-memory tiles: K tile by K tile, in it the share of each CTA of a pair (b_rows rows), in that the heads and then
// the tails, so that a CTA's part of a K tile is one contiguous run.  Also clears the status word, if given.
__global__ void linear_prepare_kernel(const float* __restrict__ B, int K, long long ldb, long long incb,
                                      const float* __restrict__ B2, int K2, long long ldb2, long long incb2, int N, int Npad,
                                      int Kpad1, int Kpad,
                                      int b_rows, float* __restrict__ out, int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && status != nullptr) *status = 0;
  if (i >= Npad * Kpad) return;
  const int n = i / Kpad, kk = i - n * Kpad;
  float v = 0.f;
  if (n < N) {
    if (kk < Kpad1) {
      if (kk < K) v = B[(long long)n * ldb + kk * incb];
    } else if (kk - Kpad1 < K2) {
      v = B2[(long long)n * ldb2 + (kk - Kpad1) * incb2];
    }
  }
  float hi, lo;
  split_tf32(v, hi, lo);
  const int share = n / b_rows, r = n - share * b_rows, kb = kk / kLinTileK, e = kk - kb * kLinTileK;
  const size_t at = (size_t)(kb * (Npad / b_rows) + share) * 2 * b_rows * kLinTileK + r * kLinTileK + (((e >> 2) ^ (r & 7)) << 2) + (e & 3);
  out[at] = hi;
  out[at + (size_t)b_rows * kLinTileK] = lo;
}

static inline int lin_kpad(long long K) { return (int)((K + kLinTileK - 1) / kLinTileK * kLinTileK); }

// One launch over checked arguments: N <= 256 columns, <= 128 of them in chunks.  clears: whether it clears the workspace's status.
static int lin_launch(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                      int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                      int64_t ldadd, int64_t k_chunk, bool clears, void* workspace, float* C, int64_t ldc, cudaStream_t st) {
  const int Npad = (int)((N + 15) / 16 * 16);
  const int Kpad1 = lin_kpad(K), Kpad2 = lin_kpad(K2), Kpad = Kpad1 + Kpad2;
  int* status = reinterpret_cast<int*>(workspace);
  float* b = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  const int num_tiles = (int)((M + kLinTileM - 1) / kLinTileM);
  // Pairs need whole 16-row groups of B in each half; a single tile has no partner.
  const bool pair = num_tiles >= 2 && Npad % 32 == 0;
  const int b_rows = pair ? Npad / 2 : Npad;   // of B in one CTA

  linear_prepare_kernel<<<(Npad * Kpad + 255) / 256, 256, 0, st>>>(B, (int)K, ldb, incb, B2, (int)K2, ldb2, incb2, (int)N, Npad,
                                                                   Kpad1, Kpad, b_rows, b, clears ? status : nullptr);
  EXB_CUDA_OK(cudaGetLastError());

  CUtensorMap tm_a, tm_a2;
  int rc = make_tensor_map_2d_f32(&tm_a, A, (unsigned long long)K, (unsigned long long)M, (unsigned long long)lda * 4, kLinTileK, kLinTileM);
  if (rc) return rc;
  if (K2 > 0) {
    rc = make_tensor_map_2d_f32(&tm_a2, A2, (unsigned long long)K2, (unsigned long long)M, (unsigned long long)lda2 * 4, kLinTileK, kLinTileM);
    if (rc) return rc;
  } else {
    tm_a2 = tm_a;
  }

  LinParams p{};
  p.b = b; p.C = C; p.bias = bias; p.status = status; p.lib_status = status_word_ptr(); p.M = M; p.ldc = ldc; p.N = (int)N; p.Npad = Npad;
  p.kblocks1 = Kpad1 / kLinTileK; p.kblocks = Kpad / kLinTileK;
  p.num_tiles = num_tiles;
  p.addend = addend; p.ldadd = ldadd;
  p.chunk = k_chunk > 0 ? (int)(k_chunk / kLinTileK) : p.kblocks;
  p.b_slot = (unsigned)b_rows * kLinTileK * 4;
  p.stage_bytes = kLinSlotBytes + 2 * p.b_slot;
  p.stages = (int)((kLinSlots * kLinSlotBytes) / p.stage_bytes);
  if (p.stages > kLinMaxStages) p.stages = kLinMaxStages;
  unsigned cols = 32;
  while (cols < (unsigned)(2 * Npad)) cols <<= 1;
  p.tmem_cols = cols;
  const size_t dyn = (size_t)kLinSlots * kLinSlotBytes + 4 * kLinEpiGroups * 4096 + 1024;
  const bool chunked = k_chunk > 0;
  auto* kern = pair ? (chunked ? linear_tf32x3_kernel<true, true> : linear_tf32x3_kernel<false, true>)
                    : (chunked ? linear_tf32x3_kernel<true, false> : linear_tf32x3_kernel<false, false>);
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
  EXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tm_a, tm_a2, p));
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_linear_workspace_bytes(int64_t N, int64_t K, int64_t K2) {
  if (N <= 0 || K <= 0 || K2 < 0) return 256;
  const int64_t Npad = (N + 15) / 16 * 16;
  return 256 + 2 * Npad * (int64_t)(lin_kpad(K) + lin_kpad(K2)) * 4;
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
  EXB_REQUIRE(k_chunk >= 0 && k_chunk % kLinTileK == 0, "linear_forward: k_chunk must be a multiple of 32");
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
  if (k_chunk == 0) return lin_launch(A, M, K, lda, B, ldb, incb, A2, K2, lda2, B2, ldb2, incb2, N, bias, addend, ldadd, 0, true, workspace, C, ldc, st);
  for (int64_t n0 = 0; n0 < N; n0 += kLinChunkedCols) {
    const int rc = lin_launch(A, M, K, lda, B + n0 * ldb, ldb, incb, A2, K2, lda2, K2 ? B2 + n0 * ldb2 : nullptr, ldb2, incb2,
                              N - n0 < kLinChunkedCols ? N - n0 : kLinChunkedCols, bias ? bias + n0 : nullptr, addend ? addend + n0 : nullptr,
                              ldadd, k_chunk, n0 == 0, workspace, C + n0, ldc, st);
    if (rc) return rc;
  }
  return EXB_OK;
}

}  // extern "C"

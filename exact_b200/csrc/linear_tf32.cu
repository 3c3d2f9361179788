// Dense layer GEMM with tf32 heads and tails in one chain per output: the products of a training forward pass whose results are
// quantised as they are, without a projection (linear_gemm.cu has the interface, the rule and the kernel of all other products).
// A saved activation's codes follow the last bits of these products.  With the other kernel's rounding, which is the closer one to
// fp64 (1.1e-7 against 1.8e-6 at 256 columns), eight codes of the 43 million of a 169,343 x 256 activation at 2 bits fall on the other
// side, and the gradients of a run differ by 0.6e-3 to 2.6e-3 from those of earlier versions at the same seed; this one keeps them.
//
// Arithmetic.  Every fp32 operand is split into a tf32 head and a tf32 tail,
//     a = a_hi + a_lo,   a_hi = rna_tf32(a),   a_lo = rna_tf32(a - a_hi)      (|a_lo| <= 2^-11 |a|),
// and the product is accumulated in fp32 as  a_hi b_hi + a_lo b_hi + a_hi b_lo.  The dropped terms
// (a_lo b_lo and the rounding of the tails) are below 2^-21 |a b|, the size of the rounding of an fp32 product; the error is that of the
// accumulator, which truncates at every MMA: 3e-7 .. 4.4e-6 (Frobenius, against fp64) at 33 to 602 columns, where a plain
// fp32 GEMM has 9e-8 .. 4.4e-7.  Non-finite inputs stay non-finite and confined to their
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
// Measured (us, here | the other kernel): 169,343 x 128 -> 256: 67 | 66, 256 -> 256: 95 | 93, 256 -> 40: 58 | 56; 2,449,029 x 256 -> 47: 683 | 574.
// The weight is split, padded and laid out as the tiles once per call by a preparation kernel.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, all roles leave their loops,
// bulk copies in flight are waited for (bounded), TMEM is freed and the status word is set.
#include "exact_b200.h"
#include "tc.cuh"

namespace exb {
namespace tf32 {

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

template <bool PAIR>
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
        for (int kb = 0; kb < p.kblocks; kb++) {
          if (kb == 0) {
            buf = t & 1;
            if (!wait(smem_u32(&s_tempty[buf]), ((uint32_t)(t >> 1) & 1u) ^ 1u)) { ok = false; break; }
            tc_fence_after();
            d_tmem = tmem_base + (uint32_t)(buf * p.Npad);
            t++;
          }
          uint32_t at;
          if (!ready(at)) { ok = false; break; }
          const int s0 = st.s;
          st.next(p.stages);
          if (elected) {
            const uint64_t ahi = umma_desc_sw128(at), alo = umma_desc_sw128(at + kLinHalf), bhi = umma_desc_sw128(at + kLinSlotBytes),
                           blo = umma_desc_sw128(at + kLinSlotBytes + p.b_slot);
#pragma unroll
            for (int k4 = 0; k4 < kLinTileK / 8; k4++) {
              const uint64_t o = (uint64_t)(k4 * 2);   // 8 tf32 = 32 bytes along K inside the swizzle atom
              mma(d_tmem, alo + o, bhi + o, kb != 0 || k4 != 0);
              mma(d_tmem, ahi + o, bhi + o, 1);
            }
#pragma unroll
            for (int k4 = 0; k4 < kLinTileK / 8; k4++) mma(d_tmem, ahi + (uint64_t)(k4 * 2), blo + (uint64_t)(k4 * 2), 1);
            commit(smem_u32(&s_empty[s0]));
            if (kb + 1 == p.kblocks) commit(smem_u32(&s_tfull[buf]));
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

// One launch over checked arguments: N <= 256 columns.
int launch_linear(const float* A, int64_t M, int64_t K, int64_t lda, const float* B, int64_t ldb, int64_t incb, const float* A2, int64_t K2,
                      int64_t lda2, const float* B2, int64_t ldb2, int64_t incb2, int64_t N, const float* bias, const float* addend,
                      int64_t ldadd, void* workspace, float* C, int64_t ldc, cudaStream_t st) {
  const int Npad = (int)((N + 15) / 16 * 16);
  const int Kpad1 = lin_kpad(K), Kpad2 = lin_kpad(K2), Kpad = Kpad1 + Kpad2;
  int* status = reinterpret_cast<int*>(workspace);
  float* b = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  const int num_tiles = (int)((M + kLinTileM - 1) / kLinTileM);
  // Pairs need whole 16-row groups of B in each half; a single tile has no partner.
  const bool pair = num_tiles >= 2 && Npad % 32 == 0;
  const int b_rows = pair ? Npad / 2 : Npad;   // of B in one CTA

  linear_prepare_kernel<<<(Npad * Kpad + 255) / 256, 256, 0, st>>>(B, (int)K, ldb, incb, B2, (int)K2, ldb2, incb2, (int)N, Npad,
                                                                   Kpad1, Kpad, b_rows, b, status);
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
  p.b_slot = (unsigned)b_rows * kLinTileK * 4;
  p.stage_bytes = kLinSlotBytes + 2 * p.b_slot;
  p.stages = (int)((kLinSlots * kLinSlotBytes) / p.stage_bytes);
  if (p.stages > kLinMaxStages) p.stages = kLinMaxStages;
  unsigned cols = 32;
  while (cols < (unsigned)(2 * Npad)) cols <<= 1;
  p.tmem_cols = cols;
  const size_t dyn = (size_t)kLinSlots * kLinSlotBytes + 4 * kLinEpiGroups * 4096 + 1024;
  auto* kern = pair ? linear_tf32x3_kernel<true> : linear_tf32x3_kernel<false>;
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

}  // namespace tf32
}  // namespace exb

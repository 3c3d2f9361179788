// Weight gradient of a quantised linear layer straight from the packed activation:
//     G[O, k] = g^T [O x N] . dequantise(packed) [N x k]
// the product grad_output.t().mm(input) of linear_backward (exact/exact/cpp_extension/backward_func.cc:87)
// with `input` still in the form qlinear.forward saved it (exact/exact/ops.py:149-154), so that the chain
// dequantize_activation -> mm of ops.py:164-169 needs neither the [N, k] fp32 activation in HBM nor a
// second pass over g.  Up to two packed activations (the two inputs of a GraphSAGE layer, which share g:
// layers.py:163-170) are multiplied in one pass; the result holds their column blocks side by side.  The
// caller applies the transposed projection to the small result: (g^T Xq) R^T.
//
// Shape of the work.  N is the number of nodes (up to millions), O <= 256, k <= 256 per pass: 2 N O k flop against
// 4 N O bytes of g, so up to about 128 columns the kernel is bound by reading g once and beyond by the tf32
// MMAs (169,343 x 256 outputs x 256 columns: 100 us at INT2, 172 us at INT8; unpacked and through the library's fp32
// GEMM: 480 us).  The contraction runs over node rows, which are the slow dimension of both operands in memory,
// while the MMA wants the contraction dimension contiguous in shared memory (K-major tiles):
//   A = g^T   [32 rows x O] boxes of g arrive by TMA (no swizzle) in a ring of raw stages; four converter
//             warps transpose them: a thread reads one output column of the box (conflict-free: the 32
//             lanes read 32 consecutive words of a row) and writes the 32 node rows of that output as one
//             128-byte row of the 128-byte-swizzled K-major tile (eight 16-byte stores);
//   B = Xq    is produced K-major by four warps that read the packed bytes (one byte = 8/bits consecutive
//             node rows of one column, which is one 16-byte chunk of the tile at INT2) and the bf16 row
//             statistics, dequantise (code / scale + min) and store to the swizzled tile.  A stage's packed
//             bytes are one contiguous run and arrive with the box of g (untiled bulk copy of the 16-byte
//             window around them), so a thread that owns a column finds them in shared memory whatever the
//             width and the number of bits; activations of more than 256 columns are multiplied in passes
//             of 256 and read their bytes from global memory.
// A tile whose contraction dimension is the slow one (MN-major) could be fed to tcgen05.mma directly by
// setting the transpose bit of the instruction descriptor; with tf32 operands and the 128-byte swizzle that
// TMA writes the unit returned zeros on this hardware, hence the transposition in shared memory.
// Converters and producers work in two pairs of warps each, which take alternate stages: a stage is a chain of waits,
// shared-memory reads, conversions and stores whose latency one group of four could not hide behind the next one
// (2,449,029 x 256 outputs, k = 32 + 32: 654 us in one group, 521 us with the producers in pairs and the boxes of g six
// stages ahead in L2, 473 us with the converters in pairs as well = 5.4 TB/s).
// Each CTA owns a contiguous range of 32-row blocks and accumulates its partial G in TMEM over the whole
// range (split over node rows across the SMs); partials go to the workspace and a second kernel adds them
// in a fixed order, so the result does not depend on timing.  tf32 inputs, fp32 accumulation: about 5e-4
// relative on G, far below the quantisation noise of the activation it is computed from.
//
// Every mbarrier wait is bounded; on expiry the CTA abandons its range, frees TMEM and raises the status words.
#include <mutex>

#include "exact_b200.h"
#include "partial_sums.cuh"
#include "tc.cuh"

namespace exb {

constexpr int kGwRows = 32;          // node rows per pipeline stage (= the K extent of a stage)
constexpr int kGwThreads = 320;      // warp 0 TMA, warp 1 MMA, warps 2-5 producers of B and epilogue, 6-9 converters
constexpr int kGwMaxStages = 6;
constexpr int kGwMaxSeg = 2;
constexpr int kGwArrivals = 4;       // warps that work on one stage: a pair of producers and a pair of converters
constexpr int kGwPrefetch = 6;       // boxes of g requested into L2 ahead of their load (the raw ring holds two to four)

struct GwSegment {
  const uint8_t* packed;
  const uint16_t* scale_bf16;
  const uint16_t* min_bf16;
  int k;        // columns of this packed activation that the pass multiplies
  int pitch;    // bytes from one row of the packed stream to the next (its width)
  int col0;     // first column of its block in the result
  unsigned smem_off;         // place of its bytes in a raw stage
  unsigned long long bytes;  // bytes of the stream from `packed` on that may be copied in 16-byte windows; 0: read from global
};

struct GwParams {
  GwSegment seg[kGwMaxSeg];
  int nseg;
  float* partial;     // [grid, Opad, kpad]
  int* lib_status;
  long long N;
  int O, Opad, kpad, bits;
  int mtiles;         // Opad / 128
  long long kblocks;  // ceil(N / 32)
  int raw_stages, stages;
  unsigned raw_bytes;                    // one raw stage: 32 rows x O fp32 of g, then the packed bytes of each activation
  int col_slots;                         // columns that the 128 producer threads take at a time (16 .. 128)
  unsigned a_bytes, b_bytes, stage_bytes, tmem_cols;
};

__device__ __forceinline__ void gw_fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// The 16-byte window of a stream that holds packed rows grp .. grp + groups - 1; bytes = 0 where they are read from
// global memory instead (a pass over part of the columns, or the end of the stream).
struct GwWindow { unsigned long long start; uint32_t bytes, skip; };
__device__ __forceinline__ GwWindow gw_window(const GwSegment& sg, long long grp, int groups) {
  const unsigned long long b0 = (unsigned long long)grp * sg.pitch, b1 = b0 + (unsigned long long)groups * sg.pitch;
  GwWindow w;
  w.start = b0 & ~15ull;
  w.skip = (uint32_t)(b0 - w.start);
  const unsigned long long end = (b1 + 15ull) & ~15ull;
  w.bytes = end <= sg.bytes ? (uint32_t)(end - w.start) : 0u;
  return w;
}

// Packed byte q of a column (its rows q * WPT .. of the stage) dequantised into the column's row of the K-major B tile:
// element r is word r % 4 of the 16-byte chunk (r / 4) ^ (column % 8).  Codes as quantization_cuda_kernel.cu:179-183
// (code / scale + min), as code * (1 / scale) + min.
template <int BITS>
__device__ __forceinline__ void gw_byte(uint32_t byte, int q, const float* inv_s, const float* min_s, uint8_t* row, int swz) {
  constexpr int WPT = 8 / BITS;
  constexpr uint32_t MASK = (1u << BITS) - 1u;
  const int r = q * WPT;
  if constexpr (WPT >= 4) {
#pragma unroll
    for (int h = 0; h < WPT / 4; h++) {
      const float4 is = *reinterpret_cast<const float4*>(inv_s + r + 4 * h), mn = *reinterpret_cast<const float4*>(min_s + r + 4 * h);
      float4 v;
      v.x = __fmaf_rn((float)((byte >> ((4 * h + 0) * BITS)) & MASK), is.x, mn.x);
      v.y = __fmaf_rn((float)((byte >> ((4 * h + 1) * BITS)) & MASK), is.y, mn.y);
      v.z = __fmaf_rn((float)((byte >> ((4 * h + 2) * BITS)) & MASK), is.z, mn.z);
      v.w = __fmaf_rn((float)((byte >> ((4 * h + 3) * BITS)) & MASK), is.w, mn.w);
      *reinterpret_cast<float4*>(row + ((((r >> 2) + h) ^ swz) << 4)) = v;
    }
  } else {
    uint8_t* dst = row + (((r >> 2) ^ swz) << 4) + (r & 3) * 4;
    float v[WPT];
#pragma unroll
    for (int x = 0; x < WPT; x++) v[x] = __fmaf_rn((float)((byte >> (x * BITS)) & MASK), inv_s[r + x], min_s[r + x]);
    if (WPT == 2) *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[WPT > 1 ? 1 : 0]);
    else *reinterpret_cast<float*>(dst) = v[0];
  }
}

// The NQ bytes of a column that one thread takes (every slices-th from `slice` on, slices = GROUPS / NQ), from shared memory.
template <int BITS, int NQ>
__device__ __forceinline__ void gw_column(uint32_t from, uint32_t pitch, int slice, long long groups_left, const float* inv_s,
                                          const float* min_s, uint8_t* row, int swz) {
  constexpr int GROUPS = kGwRows * BITS / 8;
  constexpr int SLICES = GROUPS / NQ;       // (GROUPS = 4 leaves half of eight slices without a byte)
  constexpr int kBatch = NQ < 8 ? NQ : 8;
  if (slice >= SLICES) return;
#pragma unroll
  for (int i0 = 0; i0 < NQ; i0 += kBatch) {
    uint32_t byte[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; i++)
      asm volatile("ld.shared.u8 %0, [%1];" : "=r"(byte[i]) : "r"(from + (uint32_t)(slice + (i0 + i) * SLICES) * pitch));
#pragma unroll
    for (int i = 0; i < kBatch; i++) {
      const int q = slice + (i0 + i) * SLICES;
      gw_byte<BITS>(q < groups_left ? byte[i] : 0u, q, inv_s, min_s, row, swz);
    }
  }
}

// Places of one block of 32 rows in both rings.
struct GwStages {
  RingStage raw, mma;
  __device__ __forceinline__ GwStages(const GwParams& p, int n) { skip(p, n); }
  __device__ __forceinline__ void skip(const GwParams& p, int n) {
    for (int i = 0; i < n; i++) {
      raw.next(p.raw_stages);
      mma.next(p.stages);
    }
  }
};

template <int BITS>
__global__ void __launch_bounds__(kGwThreads, 1)
grad_weight_kernel(const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ GwParams p) {
  constexpr int WPT = 8 / BITS;
  constexpr int GROUPS = kGwRows / WPT;     // packed bytes per column and stage
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long s_rfull[kGwMaxStages];    // raw box of g landed
  __shared__ __align__(8) unsigned long long s_rempty[kGwMaxStages];   // raw box transposed
  __shared__ __align__(8) unsigned long long s_full[kGwMaxStages];     // A^T and B of an MMA stage written
  __shared__ __align__(8) unsigned long long s_empty[kGwMaxStages];    // MMA stage read by the tensor core
  __shared__ __align__(8) unsigned long long s_done;
  // row statistics of the stage a producer warp works on and of the next one: a private copy per warp, so the
  // producers need no barrier among themselves
  __shared__ __align__(16) float s_scale[2][4][kGwMaxSeg][kGwRows];
  __shared__ __align__(16) float s_min[2][4][kGwMaxSeg][kGwRows];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* tiles_ptr = smem_raw + (tiles_base - smem_u32(smem_raw));
  // layout of the dynamic shared memory: raw ring, then the MMA stages (A^T tiles, B tile)
  const uint32_t mma_off = (uint32_t)p.raw_stages * p.raw_bytes;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < p.raw_stages; s++) {
      mbar_init(smem_u32(&s_rfull[s]), 1);    // the TMA thread's bytes
      mbar_init(smem_u32(&s_rempty[s]), kGwArrivals);
    }
    for (int s = 0; s < p.stages; s++) {
      mbar_init(smem_u32(&s_full[s]), kGwArrivals);
      mbar_init(smem_u32(&s_empty[s]), 1);    // tcgen05.commit
    }
    mbar_init(smem_u32(&s_done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(&s_tmem_base), p.tmem_cols);
  // B rows that hold no column of any activation stay zero for the whole kernel
  for (int s = 0; s < p.stages; s++) {
    uint4* b = reinterpret_cast<uint4*>(tiles_ptr + mma_off + (size_t)s * p.stage_bytes + p.a_bytes);
    for (unsigned i = threadIdx.x; i < p.b_bytes / 16; i += kGwThreads) b[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  gw_fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;

  // this CTA's range of 32-row blocks
  const long long per = (p.kblocks + gridDim.x - 1) / gridDim.x;
  const long long kb0 = (long long)blockIdx.x * per;
  const long long kb1 = kb0 + per < p.kblocks ? kb0 + per : p.kblocks;
  const long long nblk = kb1 > kb0 ? kb1 - kb0 : 0;

  if (warp == 0) {
    // ---------------- TMA producer: raw boxes of g ----------------
    if (lane == 0) {
      bool ok = true;
      long long it = 0;
      RingStage st;
      for (; it < nblk && ok; it++, st.next(p.raw_stages)) {
        const int s = st.s;
        const uint32_t ph = st.ph;
        if (!mbar_wait(smem_u32(&s_rempty[s]), ph ^ 1u, abort_flag)) { ok = false; break; }
        const uint32_t full = smem_u32(&s_rfull[s]);
        const uint32_t dst = tiles_base + (uint32_t)s * p.raw_bytes;
        uint32_t bytes = (uint32_t)(kGwRows * p.O * 4);
        for (int sg = 0; sg < p.nseg; sg++) bytes += gw_window(p.seg[sg], (kb0 + it) * GROUPS, GROUPS).bytes;
        mbar_arrive_expect_tx(full, bytes);
        if (it + kGwPrefetch < nblk) tma_prefetch_2d(&tm_g, 0, (int)((kb0 + it + kGwPrefetch) * kGwRows));
        tma_load_2d(dst, &tm_g, 0, (int)((kb0 + it) * kGwRows), full);
        for (int sg = 0; sg < p.nseg; sg++) {
          const GwWindow w = gw_window(p.seg[sg], (kb0 + it) * GROUPS, GROUPS);
          if (w.bytes)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             dst + p.seg[sg].smem_off),
                         "l"(p.seg[sg].packed + w.start), "r"(w.bytes), "r"(full)
                         : "memory");
        }
      }
      if (!ok) {   // leave no bulk copy in flight
        const long long t0 = clock64();
        for (int j = 0; j < p.raw_stages && j < it; j++) {
          const long long jt = it - 1 - j;
          const uint32_t bar = smem_u32(&s_rfull[jt % p.raw_stages]);
          const uint32_t ph = (uint32_t)(jt / p.raw_stages) & 1u;
          while (!mbar_try_wait(bar, ph) && clock64() - t0 < kWaitLimitCycles) {}
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_tf32(128, p.kpad);
      bool ok = true;
      RingStage st;
      for (long long it = 0; it < nblk && ok; it++, st.next(p.stages)) {
        const int s = st.s;
        const uint32_t ph = st.ph;
        if (!mbar_wait(smem_u32(&s_full[s]), ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = tiles_base + mma_off + (uint32_t)s * p.stage_bytes;
        const uint64_t b_desc = umma_desc_sw128(a_addr + p.a_bytes);
        for (int mt = 0; mt < p.mtiles; mt++) {
          const uint64_t a_desc = umma_desc_sw128(a_addr + (uint32_t)mt * (128 * 128));
#pragma unroll
          for (int k8 = 0; k8 < kGwRows / 8; k8++)   // 8 tf32 = 32 bytes along the 128-byte rows of both tiles
            umma_tf32(tmem_base + (uint32_t)(mt * p.kpad), a_desc + (uint64_t)(k8 * 2), b_desc + (uint64_t)(k8 * 2), idesc,
                      (it | k8) != 0);
        }
        umma_commit(smem_u32(&s_empty[s]));
      }
      if (ok) umma_commit(smem_u32(&s_done));
    }
  } else if (warp >= 6) {
    // ---------------- converters (warps 6..9): raw box [32 rows x O] -> A^T tiles [128 outputs x 32 rows] ----------------
    const int pair = (warp - 6) >> 1, t = threadIdx.x - 192 - pair * 64;   // output modulo 64
    GwStages st(p, pair);
    for (long long it = pair; it < nblk; it += 2, st.skip(p, 2)) {
      const int rs = st.raw.s, s = st.mma.s;
      const uint32_t rph = st.raw.ph, ph = st.mma.ph;
      // the same outcome in every lane, so that a warp leaves the loop as a whole
      // The stage first: a pair meets a place of an odd ring in every second round, which a parity alone does not tell apart; the
      // block that used the stage before has been consumed, so the one that used the raw place before (no later) has landed.
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[s]), ph ^ 1u, abort_flag))) break;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_rfull[rs]), rph, abort_flag))) break;
      const float* raw = reinterpret_cast<const float*>(tiles_ptr + (size_t)rs * p.raw_bytes);
      uint8_t* at = tiles_ptr + mma_off + (size_t)s * p.stage_bytes;
      for (int o = t; o < p.Opad; o += 64) {
        float v[kGwRows];
#pragma unroll
        for (int n = 0; n < kGwRows; n++) v[n] = o < p.O ? raw[n * p.O + o] : 0.f;
        uint8_t* row = at + (size_t)o * 128;
#pragma unroll
        for (int c = 0; c < kGwRows / 4; c++)
          *reinterpret_cast<float4*>(row + ((c ^ (o & 7)) << 4)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
      gw_fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&s_rempty[rs]));
        mbar_arrive(smem_u32(&s_full[s]));
      }
    }
  } else {
    // ---------------- producers of B = dequantised activation (warps 2..5), then the epilogue ----------------
    const int t = threadIdx.x - 64;            // 0 .. 127
    bool ok = true;
    // A thread owns every col_slots-th column (of both activations, one after the other) and, where the columns leave
    // threads over, every slices-th byte of it.
    const int grp_id = t >> 6, tt = t & 63;
    const int cslot = tt % p.col_slots, slice = tt / p.col_slots, slices = 64 / p.col_slots;
    const int ktot = p.seg[0].k + (p.nseg > 1 ? p.seg[1].k : 0);
    const int sg0 = cslot >= p.seg[0].k ? 1 : 0, j0 = cslot - (sg0 ? p.seg[0].k : 0);
    const int pw = warp - 2;                   // producer warp 0 .. 3
    // Row statistics are requested one stage ahead into registers (lane = row), turned into
    // 1 / scale (so that a code is dequantised with one FMA; a constant row has scale = inf and reciprocal 0,
    // its codes are 0 anyway) and min in this warp's shared-memory copy when their stage begins.  Rows past N
    // get 0, 0.
    // (the loaded values are not touched before their stage begins: a warp issues in order, and the first
    // instruction that needs a load result would make it wait for the load)
    uint16_t scale_next[kGwMaxSeg], min_next[kGwMaxSeg];
    auto load_stats = [&](long long it) {
      const long long n = (kb0 + it) * kGwRows + lane;
#pragma unroll
      for (int sg = 0; sg < kGwMaxSeg; sg++) {
        scale_next[sg] = 0x7f80;               // scale = inf, min = 0: reciprocal 0
        min_next[sg] = 0;
        if (sg < p.nseg && n < p.N) {
          scale_next[sg] = __ldg(p.seg[sg].scale_bf16 + n);
          min_next[sg] = __ldg(p.seg[sg].min_bf16 + n);
        }
      }
    };
    if (grp_id < nblk) load_stats(grp_id);
    GwStages st(p, grp_id);
    for (long long it = grp_id; it < nblk && ok; it += 2, st.skip(p, 2)) {
      const int rs = st.raw.s, s = st.mma.s;
      const uint32_t rph = st.raw.ph, ph = st.mma.ph;
      const int sb = (int)((it >> 1) & 1);
#pragma unroll
      for (int sg = 0; sg < kGwMaxSeg; sg++) {
        if (sg < p.nseg) {
          s_scale[sb][pw][sg][lane] = __frcp_rn(bf16_bits_to_f32(scale_next[sg]));
          s_min[sb][pw][sg][lane] = bf16_bits_to_f32(min_next[sg]);
        }
      }
      __syncwarp();                           // this warp's copy of the stage's statistics is in shared memory
      if (it + 2 < nblk) load_stats(it + 2);
      // the same outcome in every lane, so that a warp leaves the loop as a whole
      // the stage first: see the converters
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[s]), ph ^ 1u, abort_flag))) { ok = false; break; }
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_rfull[rs]), rph, abort_flag))) { ok = false; break; }
      uint8_t* btile = tiles_ptr + mma_off + (size_t)s * p.stage_bytes + p.a_bytes;
      const long long grp0 = (kb0 + it) * GROUPS;
      const long long groups_left = (p.N + WPT - 1) / WPT - grp0;
      // first column of the thread: its place was worked out before the loop (a producer warp has an SM sub-partition
      // to itself, so every dependent instruction here costs its full latency)
      int sg = sg0, j = j0;
      for (int c = cslot; c < ktot;) {
        const GwSegment& seg = p.seg[sg];
        const unsigned long long b0 = (unsigned long long)grp0 * (unsigned)seg.pitch;
        const bool windowed = ((b0 + (unsigned)(GROUPS * seg.pitch) + 15ull) & ~15ull) <= seg.bytes;
        const uint32_t from = tiles_base + (uint32_t)rs * p.raw_bytes + seg.smem_off + ((uint32_t)b0 & 15u) + (uint32_t)j;
        const int jb = seg.col0 + j;           // row of the B tile
        const float *inv_s = &s_scale[sb][pw][sg][0], *min_s = &s_min[sb][pw][sg][0];
        uint8_t* row = btile + jb * 128;
        if (windowed) {
          switch (slices) {
            case 1: gw_column<BITS, GROUPS>(from, (uint32_t)seg.pitch, slice, groups_left, inv_s, min_s, row, jb & 7); break;
            case 2: gw_column<BITS, GROUPS / 2>(from, (uint32_t)seg.pitch, slice, groups_left, inv_s, min_s, row, jb & 7); break;
            case 4: gw_column<BITS, GROUPS / 4>(from, (uint32_t)seg.pitch, slice, groups_left, inv_s, min_s, row, jb & 7); break;
            default: gw_column<BITS, (GROUPS + 7) / 8>(from, (uint32_t)seg.pitch, slice, groups_left, inv_s, min_s, row, jb & 7); break;
          }
        } else {
          const uint8_t* src = seg.packed + b0 + j;
          for (int q = slice; q < GROUPS; q += slices)
            gw_byte<BITS>(q < groups_left ? (uint32_t)__ldg(src + (size_t)q * seg.pitch) : 0u, q, inv_s, min_s, row, jb & 7);
        }
        c += p.col_slots;
        sg = c >= p.seg[0].k ? 1 : 0;
        j = c - (sg ? p.seg[0].k : 0);
      }
      gw_fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&s_rempty[rs]));
        mbar_arrive(smem_u32(&s_full[s]));
      }
    }
    // ---------------- epilogue: this CTA's partial G to the workspace ----------------
    if (ok && nblk > 0) ok = __all_sync(0xffffffffu, mbar_wait<64>(smem_u32(&s_done), 0, abort_flag));
    if (ok) {
      tc_fence_after();
      const int quad = warp & 3;
      float* dst0 = p.partial + (size_t)blockIdx.x * p.Opad * p.kpad;
      for (int mt = 0; mt < p.mtiles; mt++) {
        const int o = mt * 128 + quad * 32 + lane;
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(mt * p.kpad);
        for (int c0 = 0; c0 < p.kpad; c0 += 16) {
          float v[16];
          if (nblk > 0) {
            tmem_ld16(taddr + (uint32_t)c0, v);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = 0.f;
          }
          float4* d4 = reinterpret_cast<float4*>(dst0 + (size_t)o * p.kpad + c0);
#pragma unroll
          for (int j = 0; j < 4; j++) d4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
  if (threadIdx.x == 0 && s_abort) raise_status(p.lib_status, EXB_STATUS_GRAD_WEIGHT);
}

// out[o, j] = sum over CTAs, in a fixed order, of partial[cta, o, j].
__global__ void __launch_bounds__(32 * kSumSlices) grad_weight_reduce_kernel(const float* __restrict__ partial, int ctas, int O,
                                                                             int Opad, int kpad, int ldo,
                                                                             float* __restrict__ out) {
  __shared__ float s_part[kSumSlices][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  const float a = sum_partials(partial + i, (long long)Opad * kpad, ctas, i < O * kpad, s_part);
  if (threadIdx.y == 0 && i < O * kpad) out[(size_t)(i / kpad) * ldo + i % kpad] = a;
}

// One pass: up to 256 columns of one or two activations.  a.pitch is the width of the whole stream, a.k the columns taken.
static int gw_pass(const float* g, int64_t N, int O, GwSegment a, const GwSegment* b, int bits, int grid, void* workspace,
                   float* out, int64_t ldo, cudaStream_t st) {
  float* partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
  const int wpt = 8 / bits, groups = kGwRows / wpt;
  GwParams p{};
  p.seg[0] = a;
  p.nseg = 1;
  int kpad = (a.k + 15) / 16 * 16;
  if (b != nullptr) {
    p.seg[1] = *b;
    p.seg[1].col0 = kpad;
    kpad += (b->k + 15) / 16 * 16;
    p.nseg = 2;
  }
  p.partial = partial; p.lib_status = status_word_ptr();
  p.N = N; p.O = O; p.Opad = (O + 127) / 128 * 128; p.kpad = kpad; p.bits = bits;
  p.mtiles = p.Opad / 128;
  p.kblocks = (N + kGwRows - 1) / kGwRows;
  int ktot = 0;
  unsigned raw = (unsigned)(kGwRows * O * 4);
  for (int i = 0; i < p.nseg; i++) {
    GwSegment& s = p.seg[i];
    ktot += s.k;
    s.smem_off = raw;
    const bool whole = s.k == s.pitch && (reinterpret_cast<uintptr_t>(s.packed) & 15) == 0;
    s.bytes = whole ? (unsigned long long)((N + wpt - 1) / wpt) * (unsigned long long)s.pitch & ~15ull : 0;
    if (whole) raw += (unsigned)((groups * s.pitch + 16 + 15) & ~15);   // a window is up to 15 bytes longer at either end
  }
  p.col_slots = 16;
  while (p.col_slots < 64 && p.col_slots < ktot) p.col_slots <<= 1;
  p.raw_bytes = (raw + 1023u) & ~1023u;
  p.a_bytes = (unsigned)(p.mtiles * 128 * 128);             // one [128 x 32] fp32 tile per M tile
  p.b_bytes = (unsigned)(kpad * 128);
  p.stage_bytes = (p.a_bytes + p.b_bytes + 1023u) & ~1023u;
  // two MMA stages are enough to keep the tensor core fed; the rest of the shared memory holds raw stages in
  // flight from HBM
  constexpr long long kRoom = 216 * 1024;
  int stages = 2;
  int raw_stages = (int)((kRoom - (long long)stages * p.stage_bytes) / p.raw_bytes);
  if (raw_stages > kGwMaxStages) raw_stages = kGwMaxStages;
  EXB_REQUIRE(raw_stages >= 2, "grad_weight_from_packed: the pipeline does not fit in shared memory");
  if (raw_stages == kGwMaxStages) {
    stages = (int)((kRoom - (long long)raw_stages * p.raw_bytes) / p.stage_bytes);
    if (stages > kGwMaxStages) stages = kGwMaxStages;
  }
  p.stages = stages; p.raw_stages = raw_stages;
  unsigned cols = 32;
  while (cols < (unsigned)(p.mtiles * kpad)) cols <<= 1;
  p.tmem_cols = cols;
  if (N > 0) {
    CUtensorMap tm_g;
    int rc = make_tensor_map_2d_f32(&tm_g, g, (unsigned long long)O, (unsigned long long)N, (unsigned long long)O * 4, (unsigned)O,
                                    kGwRows, /*swizzle128=*/false);
    if (rc) return rc;
    const size_t dyn = (size_t)raw_stages * p.raw_bytes + (size_t)stages * p.stage_bytes + 1024;
#define EXB_GW_LAUNCH(BITS_)                                                                                  \
  {                                                                                                           \
    EXB_CUDA_OK(cudaFuncSetAttribute(grad_weight_kernel<BITS_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)); \
    grad_weight_kernel<BITS_><<<(unsigned)grid, kGwThreads, dyn, st>>>(tm_g, p);                              \
  }
    switch (bits) {
      case 1: EXB_GW_LAUNCH(1) break;
      case 2: EXB_GW_LAUNCH(2) break;
      case 4: EXB_GW_LAUNCH(4) break;
      default: EXB_GW_LAUNCH(8) break;
    }
#undef EXB_GW_LAUNCH
    EXB_CUDA_OK(cudaGetLastError());
  }
  const int total = O * kpad;
  grad_weight_reduce_kernel<<<(total + 31) / 32, dim3(32, kSumSlices), 0, st>>>(partial, N > 0 ? grid : 0, O, p.Opad, kpad,
                                                                                (int)ldo, out);
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

}  // namespace exb

using namespace exb;

extern "C" {

int64_t exact_grad_weight_workspace_bytes(int64_t O, int64_t k_total_padded, int max_ctas) {
  if (O <= 0 || k_total_padded <= 0 || max_ctas <= 0) return 256;
  const int64_t Opad = (O + 127) / 128 * 128;
  return 256 + (int64_t)max_ctas * Opad * k_total_padded * 4;
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
  EXB_REQUIRE(N / kGwRows < 2147483647LL, "grad_weight_from_packed: too many rows");
  cudaStream_t st = (cudaStream_t)stream;
  const long long kblocks = (N + kGwRows - 1) / kGwRows;
  long long grid = sm_count();
  if (grid > kblocks) grid = kblocks > 0 ? kblocks : 1;
  const int64_t kpass = kpad < 256 ? kpad : 256;
  const int Opad = (int)((O + 127) / 128 * 128);
  EXB_REQUIRE(workspace_bytes >= 256 + grid * (int64_t)Opad * kpass * 4,
              "grad_weight_from_packed: workspace of %lld bytes is too small (%lld needed)", (long long)workspace_bytes,
              (long long)(256 + grid * (int64_t)Opad * kpass * 4));
  const GwSegment s0{packed0, scale0, min0, (int)k0, (int)k0, 0, 0, 0}, s1{packed1, scale1, min1, (int)k1, (int)k1, 0, 0, 0};
  if (kpad <= 256) return gw_pass(g, N, (int)O, s0, k1 > 0 ? &s1 : nullptr, bits, (int)grid, workspace, out, ldo, st);
  // both activations do not fit one accumulator: each in passes of up to 256 of its columns
  for (int i = 0; i < (k1 > 0 ? 2 : 1); i++) {
    const GwSegment& s = i ? s1 : s0;
    for (int c = 0; c < s.k; c += 256) {
      GwSegment part = s;
      part.packed += c;
      part.k = s.k - c < 256 ? s.k - c : 256;
      const int rc = gw_pass(g, N, (int)O, part, nullptr, bits, (int)grid, workspace, out + (i ? k0pad : 0) + c, ldo, st);
      if (rc) return rc;
    }
  }
  return EXB_OK;
}

}  // extern "C"

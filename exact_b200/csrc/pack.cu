// Per-row stochastic quantise + bit-pack of saved activations, and unpack + dequantise.
//
// Replaces, behind a C ABI:
//   pack_single_precision    exact/exact/cpp_extension/quantization.cc:37-48,
//                            quantization_cuda_kernel.cu:63-155
//   unpack_single_precision  quantization.cc:50-62, quantization_cuda_kernel.cu:158-229
//   the torch glue around them in exact/exact/ops.py:20-98 (row min/max, scale, bf16 statistics),
//   which the fused entry point folds into the same pass over the activation.
//
// Work decomposition.  The packed stream stores, for column d, the codes of `8/bits` consecutive rows
// in one byte at (n / (8/bits)) * D + d.  An 8-row tile therefore covers whole bytes for every bit
// width.  `tpt` threads own one tile; each thread keeps 8 rows x V chunks x VEC columns in registers,
// so bytes are assembled thread-locally and stored VEC at a time, and the activation is read from
// HBM exactly once.  Row min/max go through redux.sync (folded shuffles when tpt < 32) and, when a
// tile spans several warps, a double-buffered shared-memory exchange with named barriers.  While a
// tile is processed, the next one (a contiguous run of 8*D elements) is pulled into L2 with one
// cp.async.bulk.prefetch.  The arithmetic uses the paired fp32 instructions of sm_100 (two elements per issue slot,
// each rounded exactly like the scalar instruction).
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "exact_b200.h"

namespace exb {

struct PackParams {
  const void* x;          // [N, D] fp32 or bf16 bits
  const float* noise;     // [N, D] supplied U[0,1) noise, or null -> Philox
  const float* mn_in;     // [N] caller-computed row min (reference-signature entry only)
  const float* scale_in;  // [N] caller-computed row scale (reference-signature entry only)
  uint8_t* packed;        // [ceil(N/(8/bits)) * D]
  uint16_t* scale_bf16;   // [N] or null
  uint16_t* min_bf16;     // [N] or null
  float* scale_f32;       // [N] or null
  float* min_f32;         // [N] or null
  long long N, D, ldx;    // ldx: pitch of x in elements
  long long row_offset;   // global index of row 0 (multiple of 8): keys the noise for row-sharded runs
  int tpt;                // threads per 8-row tile
  uint32_t off_lo, off_hi;
  PhiloxKey key;
};

constexpr int kMaxWarpsPerTile = 8;
constexpr int kMaxGroupsPerCta = 2;  // tiles of more than one warp: at most two per CTA

// Barrier over the threads of one multi-warp tile group; ids are literals.
__device__ __forceinline__ void group_barrier(int grp, int nthreads) {
  if (grp == 0) named_barrier<1>(nthreads);
  else named_barrier<2>(nthreads);
}

// Per-thread view of the tiling, fixed for the whole kernel.
struct TileCtx {
  long long N, D, G, ldx;
  int tpt, grp, tl, lane, lane_base;
  bool multi;
};

struct HalfBits { uint16_t bits; };   // fp16 activations: the half arithmetic of the reference's half kernels (pack_f16.cu)

// VEC adjacent elements of a row as loaded.  16-bit types stay packed in pairs: half the registers of the widened tile, and
// their minimum and maximum are taken two at a time.
template <typename InT, int VEC>
struct Raw {
  static constexpr int kWords = (VEC + 1) / 2;
  uint32_t w[kWords];
  __device__ __forceinline__ void load(const InT* p) {
    if (VEC == 4) {
      const uint2 t = __ldcs(reinterpret_cast<const uint2*>(p));
      w[0] = t.x;
      w[kWords - 1] = t.y;
    } else if (VEC == 2) {
      w[0] = __ldcs(reinterpret_cast<const uint32_t*>(p));
    } else {
      w[0] = __ldcs(reinterpret_cast<const uint16_t*>(p));
    }
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < kWords; i++) w[i] = 0u;
  }
  static __device__ __forceinline__ float low(uint32_t v) {
    if (std::is_same<InT, HalfBits>::value) return __half2float(__ushort_as_half((unsigned short)v));
    return __uint_as_float(v << 16);
  }
  static __device__ __forceinline__ float high(uint32_t v) {
    if (std::is_same<InT, HalfBits>::value) return __half2float(__ushort_as_half((unsigned short)(v >> 16)));
    return __uint_as_float(v & 0xffff0000u);
  }
  __device__ __forceinline__ float at(int e) const { return (e & 1) ? high(w[e >> 1]) : low(w[e >> 1]); }
  static __device__ __forceinline__ uint32_t pair_min(uint32_t a, uint32_t b) {
    uint32_t r;
    if (std::is_same<InT, HalfBits>::value) asm("min.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("min.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  static __device__ __forceinline__ uint32_t pair_max(uint32_t a, uint32_t b) {
    uint32_t r;
    if (std::is_same<InT, HalfBits>::value) asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  __device__ __forceinline__ void range(float& lo, float& hi) const {
    if (VEC == 1) {
      const float v = low(w[0]);
      lo = min_nan(lo, v);
      hi = max_nan(hi, v);
      return;
    }
    const uint32_t a = VEC == 4 ? pair_min(w[0], w[kWords - 1]) : w[0], b = VEC == 4 ? pair_max(w[0], w[kWords - 1]) : w[0];
    lo = min_nan3(lo, low(a), high(a));
    hi = max_nan3(hi, low(b), high(b));
  }
};
template <int VEC>
struct Raw<float, VEC> {
  float v[VEC];
  __device__ __forceinline__ void load(const float* p) { Ld<float, VEC>::load(p, v); }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < VEC; e++) v[e] = 0.f;
  }
  __device__ __forceinline__ float at(int e) const { return v[e]; }
  __device__ __forceinline__ void range(float& lo, float& hi) const {
    if (VEC == 1) {
      lo = min_nan(lo, v[0]);
      hi = max_nan(hi, v[0]);
    } else {
#pragma unroll
      for (int e = 0; e < VEC; e += 2) {
        lo = min_nan3(lo, v[e], v[(e + 1) % VEC]);
        hi = max_nan3(hi, v[e], v[(e + 1) % VEC]);
      }
    }
  }
};

// FULL: all 8 rows of the tile exist; one 64-bit base per chunk, rows addressed by 32-bit offsets.
template <typename InT, int VEC, int V, bool FULL>
__device__ __forceinline__ void load_tile(const InT* __restrict__ x, const TileCtx& c, long long tile,
                                          const long long (&col)[V], const bool (&cvalid)[V],
                                          Raw<InT, VEC> (&xv)[8][V]) {
  const long long row0 = tile << 3;
  const int rows_valid = FULL ? 8 : c.N - row0 >= 8 ? 8 : c.N > row0 ? (int)(c.N - row0) : 0;
  const unsigned Du = (unsigned)c.ldx;
#pragma unroll
  for (int v = 0; v < V; v++) {
    const InT* __restrict__ base = x + row0 * c.ldx + col[v];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      if ((FULL || r < rows_valid) && cvalid[v]) xv[r][v].load(base + r * Du);
      else xv[r][v].clear();
    }
  }
}

// Four (two, one) 8-bit codes -> one word with a code per byte.
template <int VEC>
__device__ __forceinline__ uint32_t bytes_of(const uint32_t (&code)[VEC]) {
  if (VEC == 4) {
    const uint32_t t01 = __byte_perm(code[0], code[1 % VEC], 0x0040);
    const uint32_t t23 = __byte_perm(code[2 % VEC], code[3 % VEC], 0x0040);
    return __byte_perm(t01, t23, 0x5410);
  } else if (VEC == 2) {
    return __byte_perm(code[0], code[1 % VEC], 0x0040);  // bytes 2, 3 are never stored
  }
  return code[0];
}
template <int VEC>
__device__ __forceinline__ void store_bytes(uint8_t* p, uint32_t w) {
  if (VEC == 4) __stcs(reinterpret_cast<uint32_t*>(p), w);
  else if (VEC == 2) __stcs(reinterpret_cast<uint16_t*>(p), (uint16_t)w);
  else __stcs(p, (uint8_t)w);
}
template <int VEC>
__device__ __forceinline__ uint32_t load_bytes(const uint8_t* p) {
  if (VEC == 4) return __ldcs(reinterpret_cast<const uint32_t*>(p));
  if (VEC == 2) return __ldcs(reinterpret_cast<const uint16_t*>(p));
  return __ldcs(p);
}

__device__ __forceinline__ float round_to_half(float f) { return __half2float(__float2half_rn(f)); }
// half(half(x - min) * scale) of elements e and e + 1, widened: the paired half instructions round each result once, which is
// what rounding the fp32 difference and product of halves to half gives (24 >= 2 * 11 + 2 digits).
template <typename InT, int VEC>
__device__ __forceinline__ f32x2 half_scaled(const Raw<InT, VEC>& x, int e, float mn, float sc) {
  if constexpr (std::is_same<InT, HalfBits>::value) {
    const uint32_t m = (uint32_t)__half_as_ushort(__float2half_rn(mn)) * 0x10001u;
    const uint32_t s = (uint32_t)__half_as_ushort(__float2half_rn(sc)) * 0x10001u;
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(x.w[e >> 1]), "r"(m));
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(d), "r"(s));
    return f2_pack(__half2float(__ushort_as_half((unsigned short)d)), __half2float(__ushort_as_half((unsigned short)(d >> 16))));
  } else {
    return f2_pack(0.f, 0.f);
  }
}

// (2^b - 1) / (max - min) as ops.py:39 evaluates it, reciprocal(mx - mn) * (2^b - 1), in the activation's arithmetic.
template <typename InT>
__device__ __forceinline__ float scale_of(float lo, float hi, float B) {
  if (std::is_same<InT, HalfBits>::value)
    return round_to_half(__fmul_rn(round_to_half(__fdiv_rn(1.0f, round_to_half(__fsub_rn(hi, lo)))), B));
  return __fmul_rn(__frcp_rn(__fsub_rn(hi, lo)), B);
}
// How the statistics are stored: bf16 for fp32 and bf16 activations, fp16 for fp16 ones (ops.py:80-83).
template <typename InT>
__device__ __forceinline__ uint16_t stat_bits(float f) {
  if (std::is_same<InT, HalfBits>::value) return __half_as_ushort(__float2half_rn(f));
  return f32_to_bf16_bits(f);
}

// Quantise the 8 x (V*VEC) register tile with stochastic rounding and assemble the packed bytes.
// MAGIC (only with FAST, and only when every scale of the tile is a finite non-zero number): the
// rounding is done by adding 1.5 * 2^23, the code being the low byte of the sum.
template <typename InT, int BITS, int VEC, int V, bool FAST, bool MAGIC>
__device__ __forceinline__ void quantize_rows(const PackParams& p, const TileCtx& c, long long tile, int rows_valid,
                                              const long long (&col)[V], const bool (&cvalid)[V],
                                              const Raw<InT, VEC> (&xv)[8][V], const float (&mn)[8], const float (&sc)[8]) {
  constexpr bool HALF = std::is_same<InT, HalfBits>::value;
  constexpr int WPT = 8 / BITS;
  constexpr int GPT = BITS;
  const long long row0 = tile << 3;
  // quantization_cuda_kernel.cu:89: t = fma(x - mn, s, u) - 0.5 (nvcc contracts the mul+add),
  // code = rint(max(t, 0)), no upper clamp.  With true row statistics and noise in [0, 1],
  // -0.5 <= t < 2^bits + 2, so the saturating float->unsigned conversion (NaN -> 0) equals
  // max-then-convert, and so does the low byte of t + 1.5 * 2^23 whenever the scale is finite.
  const long long noise_tile = (row0 + p.row_offset) >> 3;
  const f32x2 neg_half = f2_pack(-0.5f, -0.5f);
  const f32x2 magic = f2_pack(12582912.f, 12582912.f);
  const unsigned Du = (unsigned)c.D;
#pragma unroll
  for (int v = 0; v < V; v++) {
    if (!cvalid[v]) continue;
    uint32_t acc[GPT];
#pragma unroll
    for (int g = 0; g < GPT; g++) acc[g] = 0u;
    // MAGIC and fp32 arithmetic: with Philox noise (at most 1 - 2^-9) no code exceeds 2^bits - 1, so the rows of a byte may be
    // added instead of masked and OR-ed, on the floats' bit patterns (the exponent's share of the sum lies above the low
    // byte): one multiply-add per element instead of 1.25 permutes, shifts and masks.
    constexpr bool SUM = MAGIC && !HALF && VEC >= 2;
    uint32_t sum[VEC];

    // One Philox block per 8-row tile and PAIR of columns: its 16 bytes are the noise of rows 0..7 of the
    // even and the odd column (byte 2 r + (column & 1)), 8 bits per element: u = (h + 0.5) / 256.
    constexpr int NP = (VEC + 1) / 2;
    uint32_t w[NP][4];
    const uint32_t odd = (VEC == 1) ? (uint32_t)(col[v] & 1) : 0u;
    if (FAST || p.noise == nullptr) {
      const unsigned long long q0 = (unsigned long long)(noise_tile * ((c.D + 1) >> 1) + (col[v] >> 1));
#pragma unroll
      for (int e = 0; e < NP; e++) {
        const unsigned long long q = q0 + e;
        philox4x32_10((uint32_t)q, (uint32_t)(q >> 32), p.off_lo, p.off_hi, p.key, w[e]);
      }
    }
    const float* __restrict__ nbase = FAST ? nullptr : (p.noise ? p.noise + row0 * c.D + col[v] : nullptr);

#pragma unroll
    for (int r = 0; r < 8; r++) {
      if (FAST || r < rows_valid) {
        float un[VEC];
        if (!FAST && nbase != nullptr) Ld<float, VEC>::load(nbase + r * Du, un);
        uint32_t code[VEC];
        if (VEC >= 2) {
          const f32x2 mn2 = f2_pack(mn[r], mn[r]);
          const f32x2 sc2 = f2_pack(sc[r], sc[r]);
#pragma unroll
          for (int e = 0; e < VEC; e += 2) {
            f32x2 u2;
            if (!FAST && nbase != nullptr) {
              u2 = f2_pack(un[e], un[(e + 1) % VEC]);
            } else {
              // columns e (even) and e + 1 of this thread share the block w[e / 2]
              const float f0 = u8_to_1p(w[e >> 1][r >> 1], (r & 1) * 2);
              const float f1 = u8_to_1p(w[e >> 1][r >> 1], (r & 1) * 2 + 1);
              u2 = noise8_to_unit(f2_pack(f0, f1));
            }
            f32x2 t2;
            if (HALF) {
              // Half (op) Half rounded to half each time, then fp32 (quantization_cuda_kernel.cu:89 on c10::Half)
              t2 = f2_add(f2_add(half_scaled(xv[r][v], e, mn[r], sc[r]), u2), neg_half);
            } else {
              const f32x2 a2 = f2_sub(f2_pack(xv[r][v].at(e), xv[r][v].at((e + 1) % VEC)), mn2);
              t2 = f2_add(f2_fma(a2, sc2, u2), neg_half);
            }
            float t0, t1;
            if (MAGIC) {
              t2 = f2_add(t2, magic);
              f2_unpack(t2, t0, t1);
              code[e] = __float_as_uint(t0);            // low byte = rint(t); higher bytes are dropped below
              code[(e + 1) % VEC] = __float_as_uint(t1);
            } else {
              f2_unpack(t2, t0, t1);
              code[e] = __float2uint_rn(t0);
              code[(e + 1) % VEC] = __float2uint_rn(t1);
            }
          }
        } else {
          const float u = (!FAST && nbase != nullptr) ? un[0]
                          : noise8_to_unit(u8_to_1p(w[0][r >> 1], (r & 1) * 2 + odd));
          const float x0 = xv[r][v].at(0);
          const float t = HALF ? __fsub_rn(__fadd_rn(round_to_half(__fmul_rn(round_to_half(__fsub_rn(x0, mn[r])), sc[r])), u), 0.5f)
                               : __fsub_rn(__fmaf_rn(__fsub_rn(x0, mn[r]), sc[r], u), 0.5f);
          code[0] = __float2uint_rn(t) & 0xffu;
        }
        if (SUM) {
#pragma unroll
          for (int e = 0; e < VEC; e++)
            sum[e] = r % WPT == 0 ? code[e] : sum[e] + code[e] * (1u << ((r % WPT) * BITS));
          if (r % WPT == WPT - 1) acc[r / WPT] = bytes_of<VEC>(sum);
          continue;
        }
        const uint32_t word = bytes_of<VEC>(code);
        constexpr uint32_t kOnes = 0x01010101u;
        const int sh = (r % WPT) * BITS;
        if (sh == 0) acc[r / WPT] = word;
        else acc[r / WPT] |= (word << sh) & (kOnes * ((0xffu << sh) & 0xffu));  // uint8 narrowing per byte
      }
    }

    uint8_t* __restrict__ obase = p.packed + (tile * GPT) * c.D + col[v];
#pragma unroll
    for (int g = 0; g < GPT; g++) {
      if (FAST || tile * GPT + g < c.G) store_bytes<VEC>(obase + g * Du, acc[g]);
    }
  }
}

// Minimum over the lanes of a tile of 8 or 16 lanes of the eight lo[] and the eight hi[] (maxima negated: a negation is exact,
// and -min(-a, -b) treats NaN and signed zeros as max does), folded: at each level a lane keeps the half of the values that
// one bit of its index names and hands the other half over, so 16 reductions take 14 or 15 shuffles.  redux.sync takes one
// value per instruction, once per tile of the warp: 64 columns (two tiles a warp) 179 us against 113 us for 128 columns and
// the same 128 M elements; 130 us with the folded shuffles (which at one tile a warp lose to redux, 125 against 110 us).
// tpt = 16: lane l of the tile ends with row l & 7 (maximum for l >= 8) in v0; 8: rows 2 (l & 3) in v0 and 2 (l & 3) + 1 in
// v1 (l >= 4).  All lanes of the warp take part.
__device__ __forceinline__ void reduce_rows(const float (&lo)[8], const float (&hi)[8], int tpt, int lane, float& v0, float& v1) {
  float v[8];
  int h = tpt >> 1;
  bool upper = (lane & h) != 0;
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = min_nan(upper ? -hi[i] : lo[i], __shfl_xor_sync(0xffffffffu, upper ? lo[i] : -hi[i], h));
  h >>= 1;
  upper = (lane & h) != 0;
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = min_nan(upper ? v[i + 4] : v[i], __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + 4], h));
  h >>= 1;
  upper = (lane & h) != 0;
#pragma unroll
  for (int i = 0; i < 2; i++) v[i] = min_nan(upper ? v[i + 2] : v[i], __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + 2], h));
  v0 = v[0];
  v1 = v[1];
  if (tpt > 8) {
    h >>= 1;
    upper = (lane & h) != 0;
    v0 = min_nan(upper ? v[1] : v[0], __shfl_xor_sync(0xffffffffu, upper ? v[0] : v[1], h));
  }
}

enum TileKind { TILE_SUB = 0, TILE_WARP = 1, TILE_MULTI = 2, TILE_PAIR = 3 };   // threads per tile: 8 or 16, 32, several warps, two

// Resident CTAs of 256 threads the compiler is told to leave registers for (the second launch bound).  One lets it spend up to 168
// registers on a tile's rows, which is the faster way for most classes; the exceptions (us for 80 M elements, 1 | the bound taken):
//   two warps a tile, two loads of four columns (260 - 512 columns): 128 registers keep a fourth CTA of 128 threads resident.
//     320 columns, INT2: fp32 102 | 94, bf16 111 | 98, fp16 105 | 95.  With three or four warps a tile one stays the better
//     bound (640 columns, INT8: fp32 85 | 84, fp16 82 | 93), which is why two warps are a class of their own;
//   one warp a tile, two loads of four columns, bf16 (132 - 256 columns): 200 columns, INT2 90 | 86 (fp32 78 | 80, left at one);
//   several warps, two loads of one or two columns: three.  602 columns, INT2: fp32 109 | 96 (a 16-byte spill included), fp16 100 | 105,
//     bf16 91 | 98; INT4: 102 | 97, 115 | 107, 93 | 99.
template <typename InT>
constexpr int resident_ctas(int vec, int v, int kind) {
  if (v != 2) return 1;
  if (vec == 4) return kind == TILE_PAIR || (kind == TILE_WARP && std::is_same<InT, uint16_t>::value) ? 2 : 1;
  return kind >= TILE_MULTI ? 3 : 1;
}

// FAST: the tile has all 8 rows and the noise is drawn from Philox.  Then there is no per-row
// validity test, and -- when all 8 scales are finite and non-zero, i.e. no row is constant or holds
// an infinity or a NaN -- round-to-nearest-even is done by adding 1.5 * 2^23 (the code is then the
// low byte of the float) instead of a float->int conversion.
template <typename InT, int BITS, int VEC, int V, int KIND, bool FAST>
__device__ __forceinline__ bool process_tile(const PackParams& p, const TileCtx& c, long long tile, int it,
                                             const long long (&col)[V], const bool (&cvalid)[V],
                                             const Raw<InT, VEC> (&xv)[8][V], float* s_part, float* s_fin) {
  const long long row0 = tile << 3;
  const int rows_valid = FAST ? 8 : c.N - row0 >= 8 ? 8 : c.N > row0 ? (int)(c.N - row0) : 0;   // 0: past the end, with its warp
  const float B = (float)((1 << BITS) - 1);

  // ---- row statistics ----------------------------------------------------------------------------
  float lo[8], hi[8], mn[8], sc[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    lo[r] = __int_as_float(0x7f800000);
    hi[r] = __int_as_float(0xff800000);
#pragma unroll
    for (int v = 0; v < V; v++)
      if (cvalid[v]) xv[r][v].range(lo[r], hi[r]);
    if (KIND != TILE_SUB) {
      lo[r] = redux_min_nan(lo[r], 0xffffffffu);
      hi[r] = redux_max_nan(hi[r], 0xffffffffu);
    }
  }
  bool finite = true;  // all 8 scales are finite numbers (warp-uniform)
  if (KIND < TILE_MULTI) {
    const float inf = __int_as_float(0x7f800000);
    // 0 < s < inf  <=>  the row's range is a finite non-zero number, hence every x in it is finite
    if (KIND == TILE_WARP) {
      // lane (tl & 7) turns row (tl & 7)'s range into a scale, then the group shares the 8 scales.
      const int my = c.tl & 7;
      float lo_my = lo[0], hi_my = hi[0];
#pragma unroll
      for (int r = 1; r < 8; r++) {
        lo_my = (my == r) ? lo[r] : lo_my;
        hi_my = (my == r) ? hi[r] : hi_my;
      }
      const float s_my = scale_of<InT>(lo_my, hi_my, B);
      if (FAST) finite = __all_sync(0xffffffffu, s_my > 0.f && s_my < inf);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        sc[r] = __shfl_sync(0xffffffffu, s_my, r);
        mn[r] = lo[r];
      }
    } else {
      float v0, v1;
      reduce_rows(lo, hi, c.tpt, c.lane, v0, v1);
      const int half = c.tpt >> 1;                             // the lane's partner across `half` holds the other extreme
      const float o0 = __shfl_xor_sync(0xffffffffu, v0, half), o1 = c.tpt == 8 ? __shfl_xor_sync(0xffffffffu, v1, half) : 0.f;
      const bool holds_max = (c.tl & half) != 0;
      const float lo0 = holds_max ? o0 : v0, s0 = scale_of<InT>(lo0, -(holds_max ? v0 : o0), B);
      float lo1 = 0.f, s1 = 1.f;
      if (c.tpt == 8) {
        lo1 = holds_max ? o1 : v1;
        s1 = scale_of<InT>(lo1, -(holds_max ? v1 : o1), B);
      }
      if (FAST) finite = __all_sync(0xffffffffu, s0 > 0.f && s0 < inf && s1 > 0.f && s1 < inf);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int from = c.lane_base + (c.tpt == 8 ? r >> 1 : r);
        mn[r] = __shfl_sync(0xffffffffu, c.tpt == 8 && (r & 1) ? lo1 : lo0, from);
        sc[r] = __shfl_sync(0xffffffffu, c.tpt == 8 && (r & 1) ? s1 : s0, from);
      }
    }
    // lane tl < 8 of the tile writes row tl's statistics
    if (c.tl < rows_valid) {
      float s_my = sc[0], lo_my = mn[0];
#pragma unroll
      for (int r = 1; r < 8; r++) {
        s_my = (c.tl == r) ? sc[r] : s_my;
        lo_my = (c.tl == r) ? mn[r] : lo_my;
      }
      const long long row = row0 + c.tl;
      if (p.scale_bf16) p.scale_bf16[row] = stat_bits<InT>(s_my);
      if (p.min_bf16) p.min_bf16[row] = stat_bits<InT>(lo_my);
      if (p.scale_f32) p.scale_f32[row] = s_my;
      if (p.min_f32) p.min_f32[row] = lo_my;
    }
  } else {
    float* part = s_part + ((it & 1) * kMaxGroupsPerCta + c.grp) * (kMaxWarpsPerTile * 16);
    float* fin = s_fin + ((it & 1) * kMaxGroupsPerCta + c.grp) * 16;
    const int wt = c.tl >> 5;  // warp within the tile
    const int nwt = c.tpt >> 5;
    if (c.lane == 0) {
#pragma unroll
      for (int r = 0; r < 8; r++) {
        part[wt * 16 + r] = lo[r];
        part[wt * 16 + 8 + r] = hi[r];
      }
    }
    group_barrier(c.grp, c.tpt);
    if (c.tl < 8) {
      float lo_f = part[c.tl], hi_f = part[8 + c.tl];
      for (int w = 1; w < nwt; w++) {
        lo_f = min_nan(lo_f, part[w * 16 + c.tl]);
        hi_f = max_nan(hi_f, part[w * 16 + 8 + c.tl]);
      }
      const float s_f = scale_of<InT>(lo_f, hi_f, B);
      fin[c.tl] = lo_f;
      fin[8 + c.tl] = s_f;
      if (c.tl < rows_valid) {
        const long long row = row0 + c.tl;
        if (p.scale_bf16) p.scale_bf16[row] = stat_bits<InT>(s_f);
        if (p.min_bf16) p.min_bf16[row] = stat_bits<InT>(lo_f);
        if (p.scale_f32) p.scale_f32[row] = s_f;
        if (p.min_f32) p.min_f32[row] = lo_f;
      }
    }
    group_barrier(c.grp, c.tpt);
    const float4* f = reinterpret_cast<const float4*>(fin);
    const float4 a = f[0], b = f[1], cc = f[2], d = f[3];
    mn[0] = a.x; mn[1] = a.y; mn[2] = a.z; mn[3] = a.w;
    mn[4] = b.x; mn[5] = b.y; mn[6] = b.z; mn[7] = b.w;
    sc[0] = cc.x; sc[1] = cc.y; sc[2] = cc.z; sc[3] = cc.w;
    sc[4] = d.x; sc[5] = d.y; sc[6] = d.z; sc[7] = d.w;
    if (FAST) {
      float mx_s = sc[0], mn_s = sc[0];
#pragma unroll
      for (int r = 1; r < 8; r++) {
        mx_s = max_nan(mx_s, sc[r]);
        mn_s = min_nan(mn_s, sc[r]);
      }
      finite = mn_s > 0.f && mx_s < __int_as_float(0x7f800000);
    }
  }

  // ---- quantise with stochastic rounding and assemble bytes ---------------------------------------
  // `finite` is uniform over the threads of the tile; tiles with a constant / inf / NaN row take the
  // general path, which is also the one of ragged and supplied-noise tiles.
  // `finite` is uniform over the threads of the tile.  A full Philox tile with a constant / inf / NaN
  // row is handed back to the caller, which redoes it on the general path.
  if (FAST) {
    if (!finite) return false;
    quantize_rows<InT, BITS, VEC, V, true, true>(p, c, tile, 8, col, cvalid, xv, mn, sc);
  } else {
    quantize_rows<InT, BITS, VEC, V, false, false>(p, c, tile, rows_valid, col, cvalid, xv, mn, sc);
  }
  return true;
}

template <typename InT, int BITS, int VEC, int V, int KIND>
__global__ void __launch_bounds__(256, resident_ctas<InT>(VEC, V, KIND))
quantize_pack_kernel(const __grid_constant__ PackParams p) {
  constexpr int WPT = 8 / BITS;
  __shared__ float s_part[2 * kMaxGroupsPerCta * kMaxWarpsPerTile * 16];
  __shared__ __align__(16) float s_fin[2 * kMaxGroupsPerCta * 16];

  TileCtx c;
  c.N = p.N; c.D = p.D; c.ldx = p.ldx;
  c.G = (p.N + WPT - 1) / WPT;
  c.tpt = p.tpt;
  c.grp = threadIdx.x / c.tpt;
  c.tl = threadIdx.x - c.grp * c.tpt;
  c.lane = threadIdx.x & 31;
  c.lane_base = (c.tpt < 32) ? (c.lane / c.tpt) * c.tpt : 0;
  c.multi = c.tpt > 32;
  const int tiles_per_cta = blockDim.x / c.tpt;
  const long long num_tiles = (p.N + 7) >> 3;
  const long long full_tiles = p.N >> 3;
  const long long stride = (long long)gridDim.x * tiles_per_cta;
  const InT* __restrict__ x = reinterpret_cast<const InT*>(p.x);

  long long col[V];
  bool cvalid[V];
#pragma unroll
  for (int v = 0; v < V; v++) {
    col[v] = (long long)(c.tl + v * c.tpt) * VEC;
    cvalid[v] = col[v] < p.D;
  }

  // The next tile (one contiguous run of 8 * D elements) is pulled into L2 by a single bulk-prefetch
  // instruction while the current one is processed, so the register loads of the next iteration
  // find their lines on chip.
  const long long tile_bytes = 8 * p.D * (long long)sizeof(InT);
  const bool can_prefetch = p.ldx == p.D && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0 && (tile_bytes & 15) == 0;
  const bool philox = p.noise == nullptr;
  Raw<InT, VEC> xv[8][V];
  int it = 0;
  // The tiles of a warp (several when tpt < 32) go through the loop together, past the end and on the general path too: the
  // shuffles below always have all lanes.
  const int in_warp = KIND == TILE_SUB ? c.lane / c.tpt : 0, last_in_warp = KIND == TILE_SUB ? 32 / c.tpt - 1 : 0;
  for (long long tile = (long long)blockIdx.x * tiles_per_cta + c.grp; tile - in_warp < num_tiles; tile += stride, ++it) {
    const long long next = tile + stride;
    if (c.tl == 0 && can_prefetch && next < full_tiles) {  // never the ragged last tile
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x + (next << 3) * p.D), "r"((uint32_t)tile_bytes)
                   : "memory");
    }
    bool done = false;
    if (philox && tile - in_warp + last_in_warp < full_tiles) {
      load_tile<InT, VEC, V, true>(x, c, tile, col, cvalid, xv);
      done = process_tile<InT, BITS, VEC, V, KIND, true>(p, c, tile, it, col, cvalid, xv, s_part, s_fin);
      if (!done) ++it;  // the redo below exchanges its statistics through the other shared-memory buffer
    }
    if (!done) {
      load_tile<InT, VEC, V, false>(x, c, tile, col, cvalid, xv);
      process_tile<InT, BITS, VEC, V, KIND, false>(p, c, tile, it, col, cvalid, xv, s_part, s_fin);
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// pack_single_precision with caller-computed statistics (the reference signature).  One thread per
// (8-row tile, column): any D, any alignment, and the reference's exact conversion
// __float2int_rn(fmax(t, 0)) for arbitrary caller-supplied scales.
template <typename InT, int BITS>
__global__ void __launch_bounds__(256) pack_given_stats_kernel(const __grid_constant__ PackParams p) {
  constexpr int WPT = 8 / BITS;
  constexpr int GPT = BITS;
  const InT* __restrict__ x = reinterpret_cast<const InT*>(p.x);
  const long long num_tiles = (p.N + 7) >> 3;
  const long long total = num_tiles * p.D;
  const long long G = (p.N + WPT - 1) / WPT;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long tile = idx / p.D;
    const long long d = idx - tile * p.D;
    const long long row0 = tile << 3;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (p.noise == nullptr) {
      const unsigned long long q = (unsigned long long)(((row0 + p.row_offset) >> 3) * ((p.D + 1) >> 1) + (d >> 1));
      philox4x32_10((uint32_t)q, (uint32_t)(q >> 32), p.off_lo, p.off_hi, p.key, w);
    }
    uint32_t acc[GPT];
#pragma unroll
    for (int g = 0; g < GPT; g++) acc[g] = 0u;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const long long n = row0 + r;
      if (n < p.N) {
        float xv[1];
        Ld<InT, 1>::load(x + n * p.D + d, xv);
        const float u = (p.noise != nullptr) ? __ldcs(p.noise + n * p.D + d)
                        : noise8_to_unit(u8_to_1p(w[r >> 1], (r & 1) * 2 + (uint32_t)(d & 1)));
        const float t = __fsub_rn(__fmaf_rn(__fsub_rn(xv[0], __ldg(p.mn_in + n)), __ldg(p.scale_in + n), u), 0.5f);
        const uint32_t code = (uint32_t)__float2int_rn(fmaxf(t, 0.f));  // quantization_cuda_kernel.cu:89
        acc[r / WPT] |= code << ((r % WPT) * BITS);
      }
    }
#pragma unroll
    for (int g = 0; g < GPT; g++) {
      const long long gi = tile * GPT + g;
      if (gi < G) p.packed[gi * p.D + d] = (uint8_t)acc[g];
    }
  }
}

// ---------------------------------------------------------------------------------------------------
struct UnpackParams {
  const uint8_t* packed;
  const void* scale;  // [N] fp32 or bf16 bits
  const void* mn;     // [N]
  void* out;          // [N, D], fp32 (fp16 with fp16 statistics)
  long long N, D;
  int tpt;
  int vec_stats;  // 1: scale/min are 16-byte aligned, whole-tile vector loads are legal
};

template <int VEC>
__device__ __forceinline__ void store_halves(__half* p, const float (&o)[VEC]) {
  if (VEC == 4) {
    const __half2 a = __floats2half2_rn(o[0], o[1 % VEC]), b = __floats2half2_rn(o[2 % VEC], o[3 % VEC]);
    __stcs(reinterpret_cast<uint2*>(p), make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b)));
  } else if (VEC == 2) {
    const __half2 a = __floats2half2_rn(o[0], o[1 % VEC]);
    __stcs(reinterpret_cast<uint32_t*>(p), *reinterpret_cast<const uint32_t*>(&a));
  } else {
    *p = __float2half_rn(o[0]);
  }
}

// code / s by the Markstein sequence q0 = c*r, rem = fma(-q0, s, c), q = fma(rem, r, q0) with r the
// correctly rounded reciprocal of s: equal to the IEEE quotient for every code 0..255 and every normal
// s (checked exhaustively over all 2^23 significands), used when 2^-100 <= |s| <= 2^100; any other
// scale (inf from a constant row, NaN, denormal) takes the division instruction sequence.
__device__ __forceinline__ bool scale_is_tame(float s) {
  const uint32_t e = (__float_as_uint(s) >> 23) & 0xffu;
  return e >= 27u && e <= 227u;
}

// STATS: 0 fp32, 1 bf16 (fp32 result), 2 fp16 (fp16 result, every step rounded to half: quantization_cuda_kernel.cu:182 on
// c10::Half).
template <int BITS, int VEC, int V, int STATS>
__global__ void __launch_bounds__(256)
unpack_dequant_kernel(const __grid_constant__ UnpackParams p) {
  constexpr bool STATS_BF16 = STATS == 1, HALF = STATS == 2;
  constexpr int WPT = 8 / BITS;
  constexpr int GPT = BITS;
  constexpr uint32_t MASKREP = 0x01010101u * ((1u << BITS) - 1u);
  const long long N = p.N, D = p.D;
  const int tpt = p.tpt;
  const int grp = threadIdx.x / tpt;
  const int tl = threadIdx.x - grp * tpt;
  const int lane = threadIdx.x & 31;
  const int lane_base = (tpt < 32) ? (lane / tpt) * tpt : 0;
  const unsigned gmask = (tpt < 32) ? (((1u << tpt) - 1u) << lane_base) : 0xffffffffu;
  const int tiles_per_cta = blockDim.x / tpt;
  const long long num_tiles = (N + 7) >> 3;
  const long long G = (N + WPT - 1) / WPT;
  const f32x2 neg_2p23 = f2_pack(-8388608.f, -8388608.f);

  long long col[V];
  bool cvalid[V];
#pragma unroll
  for (int v = 0; v < V; v++) {
    col[v] = (long long)(tl + v * tpt) * VEC;
    cvalid[v] = col[v] < D;
  }

  for (long long tile = (long long)blockIdx.x * tiles_per_cta + grp; tile < num_tiles;
       tile += (long long)gridDim.x * tiles_per_cta) {
    const long long row0 = tile << 3;
    const int rows_valid = (N - row0 >= 8) ? 8 : (int)(N - row0);

    uint32_t b[GPT][V];
#pragma unroll
    for (int g = 0; g < GPT; g++) {
      const long long gi = tile * GPT + g;
#pragma unroll
      for (int v = 0; v < V; v++) b[g][v] = (gi < G && cvalid[v]) ? load_bytes<VEC>(p.packed + gi * D + col[v]) : 0u;
    }

    float s[8], m[8];
    if (rows_valid == 8 && p.vec_stats) {
      if (STATS_BF16 || HALF) {
        const uint4 sv = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.scale) + row0));
        const uint4 mv = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.mn) + row0));
        const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
        const uint32_t mw[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type, 2>;
          s[2 * i] = Stat::low(sw[i]);
          s[2 * i + 1] = Stat::high(sw[i]);
          m[2 * i] = Stat::low(mw[i]);
          m[2 * i + 1] = Stat::high(mw[i]);
        }
      } else {
        const float4* sp = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.scale) + row0);
        const float4* mp = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.mn) + row0);
        const float4 s0 = __ldg(sp), s1 = __ldg(sp + 1), m0 = __ldg(mp), m1 = __ldg(mp + 1);
        s[0] = s0.x; s[1] = s0.y; s[2] = s0.z; s[3] = s0.w; s[4] = s1.x; s[5] = s1.y; s[6] = s1.z; s[7] = s1.w;
        m[0] = m0.x; m[1] = m0.y; m[2] = m0.z; m[3] = m0.w; m[4] = m1.x; m[5] = m1.y; m[6] = m1.z; m[7] = m1.w;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 8; r++) {
        if (r < rows_valid) {
          if (STATS_BF16 || HALF) {
            using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type, 1>;
            s[r] = Stat::low(__ldg(reinterpret_cast<const uint16_t*>(p.scale) + row0 + r));
            m[r] = Stat::low(__ldg(reinterpret_cast<const uint16_t*>(p.mn) + row0 + r));
          } else {
            s[r] = __ldg(reinterpret_cast<const float*>(p.scale) + row0 + r);
            m[r] = __ldg(reinterpret_cast<const float*>(p.mn) + row0 + r);
          }
        } else {
          s[r] = 1.f;
          m[r] = 0.f;
        }
      }
    }

    // one correctly rounded reciprocal per row, computed by lane (lane & 7) and shared in the group
    const int my = lane & 7;
    float s_my = s[0];
#pragma unroll
    for (int r = 1; r < 8; r++) s_my = (my == r) ? s[r] : s_my;
    const float r_my = __frcp_rn(s_my);
    const bool tame = __all_sync(gmask, scale_is_tame(s_my));
    float rcp[8];
#pragma unroll
    for (int r = 0; r < 8; r++) rcp[r] = __shfl_sync(gmask, r_my, lane_base + r);

#pragma unroll
    for (int r = 0; r < 8; r++) {
      if (r < rows_valid) {
        const int sh = (r % WPT) * BITS;
        const f32x2 r2 = f2_pack(rcp[r], rcp[r]);
        const f32x2 ns2 = f2_pack(-s[r], -s[r]);
        const f32x2 m2 = f2_pack(m[r], m[r]);
#pragma unroll
        for (int v = 0; v < V; v++) {
          if (cvalid[v]) {
            const uint32_t t = (BITS == 8) ? b[r / WPT][v] : ((b[r / WPT][v] >> sh) & MASKREP);
            float cf[VEC], o[VEC];
#pragma unroll
            for (int e = 0; e < VEC; e++)  // 0x4B0000cc = 2^23 + code
              cf[e] = __uint_as_float(__byte_perm(t, 0x4b000000u, 0x7540 | e));
            if (VEC >= 2 && tame) {
#pragma unroll
              for (int e = 0; e < VEC; e += 2) {
                const f32x2 c2 = f2_add(f2_pack(cf[e], cf[(e + 1) % VEC]), neg_2p23);
                const f32x2 q0 = f2_mul(c2, r2);
                const f32x2 rem = f2_fma(q0, ns2, c2);
                const f32x2 q = f2_fma(rem, r2, q0);
                if (HALF) {
                  float q0r, q1r;
                  f2_unpack(q, q0r, q1r);
                  f2_unpack(f2_add(f2_pack(round_to_half(q0r), round_to_half(q1r)), m2), o[e], o[(e + 1) % VEC]);
                } else {
                  f2_unpack(f2_add(q, m2), o[e], o[(e + 1) % VEC]);
                }
              }
            } else {
#pragma unroll
              for (int e = 0; e < VEC; e++)  // quantization_cuda_kernel.cu:182: IEEE division, then addition
              {
                const float q = __fdiv_rn(__fsub_rn(cf[e], 8388608.f), s[r]);
                o[e] = __fadd_rn(HALF ? round_to_half(q) : q, m[r]);
              }
            }
            if (HALF) store_halves<VEC>(static_cast<__half*>(p.out) + (row0 + r) * D + col[v], o);
            else StF32<VEC>::store(static_cast<float*>(p.out) + (row0 + r) * D + col[v], o);
          }
        }
      }
    }
  }
}

// Unpack + dequantise of an odd number of columns.  Rows then start on odd elements and the tiled kernel stores one element per
// lane; here the output is one run of elements and a thread makes four adjacent ones, whatever rows they fall into, and stores
// them together.  300,001 x 47 at INT2: 62 us in the tiled kernel (fp16 64, 42 in the plain one), 37 here.
template <int BITS, int STATS>
__global__ void __launch_bounds__(256) unpack_flat_kernel(const __grid_constant__ UnpackParams p) {
  constexpr bool HALF = STATS == 2;
  constexpr int WPT = 8 / BITS;
  constexpr uint32_t MASK = (1u << BITS) - 1u;
  const long long total = p.N * p.D;
  const uint32_t D = (uint32_t)p.D;
  for (long long i0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4; i0 < total; i0 += (long long)gridDim.x * blockDim.x * 4) {
    long long n = total < (1LL << 32) ? (long long)((uint32_t)i0 / D) : i0 / p.D;
    uint32_t d = (uint32_t)(i0 - n * p.D);
    float s = 1.f, m = 0.f, rcp = 1.f;
    bool tame = true;
    const uint8_t* src = nullptr;
    int sh = 0;
    auto row = [&]() {
      if (STATS == 0) {
        s = __ldg(reinterpret_cast<const float*>(p.scale) + n);
        m = __ldg(reinterpret_cast<const float*>(p.mn) + n);
      } else {
        using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type, 1>;
        s = Stat::low(__ldg(reinterpret_cast<const uint16_t*>(p.scale) + n));
        m = Stat::low(__ldg(reinterpret_cast<const uint16_t*>(p.mn) + n));
      }
      rcp = __frcp_rn(s);
      tame = scale_is_tame(s);
      src = p.packed + (n / WPT) * p.D;
      sh = (int)(n % WPT) * BITS;
    };
    row();
    float o[4];
#pragma unroll
    for (int x = 0; x < 4; x++) {
      o[x] = 0.f;
      if (i0 + x < total) {
        const float c = (float)((__ldg(src + d) >> sh) & MASK);
        float q;
        if (tame) {
          const float q0 = __fmul_rn(c, rcp);
          q = __fmaf_rn(__fmaf_rn(-q0, s, c), rcp, q0);
        } else {
          q = __fdiv_rn(c, s);
        }
        o[x] = __fadd_rn(HALF ? round_to_half(q) : q, m);
        if (++d == D && x < 3 && i0 + x + 1 < total) {
          d = 0;
          n++;
          row();
        }
      }
    }
    if (i0 + 4 <= total) {
      if (HALF) store_halves<4>(static_cast<__half*>(p.out) + i0, o);
      else StF32<4>::store(static_cast<float*>(p.out) + i0, o);
    } else {
      for (int x = 0; i0 + x < total; x++) {
        if (HALF) static_cast<__half*>(p.out)[i0 + x] = __float2half_rn(o[x]);
        else static_cast<float*>(p.out)[i0 + x] = o[x];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// Host side: shape -> (VEC, V, tpt, block) and launch.
struct TileShape {
  int vec, v, tpt, block;
};

static int pow2ceil(int x) {
  int p = 1;
  while (p < x) p <<= 1;
  return p;
}

// Chooses the register tiling for D columns whose accesses may use `max_vec` elements per load.
static bool choose_shape(long long D, int max_vec, TileShape* s) {
  int vec = (max_vec >= 4 && D % 4 == 0) ? 4 : (max_vec >= 2 && D % 2 == 0) ? 2 : 1;
  long long C = D / vec;
  int v, tpt;
  if (C <= 32) {
    v = 1;
    tpt = pow2ceil((int)C);
    if (tpt < 8) tpt = 8;
  } else if (C <= 64) {
    v = 2;
    tpt = 32;
  } else if (C <= 512) {
    v = 2;
    tpt = (int)(((C + 1) / 2 + 31) / 32) * 32;
  } else if (C <= 1024) {
    v = 4;
    tpt = (int)(((C + 3) / 4 + 31) / 32) * 32;
  } else {
    return false;
  }
  int block = tpt >= 128 ? tpt : tpt * (128 / tpt);
  s->vec = vec; s->v = v; s->tpt = tpt; s->block = block;
  return true;
}

template <typename K>
static int persistent_grid(K kernel, int block, long long work_ctas, int* grid) {
  int per_sm = 0;
  EXB_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0));
  if (per_sm < 1) per_sm = 1;
  long long g = (long long)sm_count() * per_sm;
  if (g > work_ctas) g = work_ctas;
  if (g < 1) g = 1;
  *grid = (int)g;
  return EXB_OK;
}

template <typename InT, int BITS>
static int launch_pack(const PackParams& p, const TileShape& s, cudaStream_t st) {
  const long long tiles = (p.N + 7) / 8;
  const int tiles_per_cta = s.block / s.tpt;
  const long long ctas = (tiles + tiles_per_cta - 1) / tiles_per_cta;
  int grid = 1;
  const int kind = s.tpt < 32 ? TILE_SUB : s.tpt == 32 ? TILE_WARP : s.tpt == 64 && s.vec == 4 ? TILE_PAIR : TILE_MULTI;
#define EXB_PACK_CASE(VEC_, V_, KIND_)                                                 \
  if (s.vec == VEC_ && s.v == V_ && kind == KIND_) {                                   \
    auto k = quantize_pack_kernel<InT, BITS, VEC_, V_, KIND_>;                         \
    int rc = persistent_grid(k, s.block, ctas, &grid);                                 \
    if (rc) return rc;                                                                 \
    k<<<grid, s.block, 0, st>>>(p);                                                    \
    EXB_CUDA_OK(cudaGetLastError());                                                   \
    return EXB_OK;                                                                     \
  }
  EXB_PACK_CASE(4, 1, TILE_SUB) EXB_PACK_CASE(4, 1, TILE_WARP) EXB_PACK_CASE(4, 2, TILE_WARP) EXB_PACK_CASE(4, 2, TILE_PAIR) EXB_PACK_CASE(4, 2, TILE_MULTI)
  EXB_PACK_CASE(4, 4, TILE_MULTI) EXB_PACK_CASE(2, 4, TILE_MULTI) EXB_PACK_CASE(1, 4, TILE_MULTI)
  EXB_PACK_CASE(2, 1, TILE_SUB) EXB_PACK_CASE(2, 1, TILE_WARP) EXB_PACK_CASE(2, 2, TILE_WARP) EXB_PACK_CASE(2, 2, TILE_MULTI)
  EXB_PACK_CASE(1, 1, TILE_SUB) EXB_PACK_CASE(1, 1, TILE_WARP) EXB_PACK_CASE(1, 2, TILE_WARP) EXB_PACK_CASE(1, 2, TILE_MULTI)
#undef EXB_PACK_CASE
  return fail(EXB_ERR_UNSUPPORTED, "no pack kernel for vec=%d v=%d", s.vec, s.v);
}

template <typename InT>
static int launch_pack_bits(const PackParams& p, int bits, const TileShape& s, cudaStream_t st) {
  switch (bits) {
    case 1: return launch_pack<InT, 1>(p, s, st);
    case 2: return launch_pack<InT, 2>(p, s, st);
    case 4: return launch_pack<InT, 4>(p, s, st);
    case 8: return launch_pack<InT, 8>(p, s, st);
  }
  return fail(EXB_ERR_ARG, "bits must be 1, 2, 4 or 8 (got %d)", bits);
}

template <typename InT>
static int launch_given_stats(const PackParams& p, int bits, cudaStream_t st) {
  const long long total = ((p.N + 7) / 8) * p.D;
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  switch (bits) {
    case 1: pack_given_stats_kernel<InT, 1><<<(int)blocks, 256, 0, st>>>(p); break;
    case 2: pack_given_stats_kernel<InT, 2><<<(int)blocks, 256, 0, st>>>(p); break;
    case 4: pack_given_stats_kernel<InT, 4><<<(int)blocks, 256, 0, st>>>(p); break;
    default: pack_given_stats_kernel<InT, 8><<<(int)blocks, 256, 0, st>>>(p); break;
  }
  EXB_CUDA_OK(cudaGetLastError());
  return EXB_OK;
}

static int align_vec(const void* ptr, int elem_bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(ptr);
  if (a % (4 * elem_bytes) == 0) return 4;
  if (a % (2 * elem_bytes) == 0) return 2;
  return 1;
}

constexpr int kDtypeHalf = 2;   // inside the library: exact_quantize_pack_f16

static int pack_common(const void* x, int dtype, long long N, long long D, long long ldx, int bits,
                       const float* noise, const float* mn_in, const float* scale_in,
                       unsigned long long seed, unsigned long long offset, long long row_offset,
                       uint8_t* packed, uint16_t* scale_bf16, uint16_t* min_bf16, float* scale_f32,
                       float* min_f32, cudaStream_t st) {
  EXB_REQUIRE(bits == 1 || bits == 2 || bits == 4 || bits == 8, "bits must be 1, 2, 4 or 8 (got %d)", bits);
  EXB_REQUIRE(dtype == EXACT_DTYPE_F32 || dtype == EXACT_DTYPE_BF16 || dtype == kDtypeHalf,
              "pack: dtype must be EXACT_DTYPE_F32 or EXACT_DTYPE_BF16 (got %d)", dtype);
  EXB_REQUIRE(N >= 0 && D >= 0, "pack: negative shape %lld x %lld", N, D);
  EXB_REQUIRE(row_offset >= 0 && row_offset % 8 == 0, "pack: row_offset must be a non-negative multiple of 8");
  if (N == 0 || D == 0) return EXB_OK;
  EXB_REQUIRE(x != nullptr && packed != nullptr, "pack: null data or output pointer");
  PackParams p;
  p.x = x; p.noise = noise; p.mn_in = mn_in; p.scale_in = scale_in;
  p.packed = packed; p.scale_bf16 = scale_bf16; p.min_bf16 = min_bf16;
  p.scale_f32 = scale_f32; p.min_f32 = min_f32;
  p.N = N; p.D = D; p.ldx = ldx; p.row_offset = row_offset; p.tpt = 0;
  p.off_lo = (uint32_t)offset; p.off_hi = (uint32_t)(offset >> 32);
  p.key = make_philox_key(seed);
  if (mn_in != nullptr) {
    if (dtype == EXACT_DTYPE_F32) return launch_given_stats<float>(p, bits, st);
    return launch_given_stats<uint16_t>(p, bits, st);
  }
  const int eb = dtype == EXACT_DTYPE_F32 ? 4 : 2;
  int max_vec = align_vec(x, eb);
  if (ldx % 4 != 0) max_vec = ldx % 2 != 0 ? 1 : max_vec < 2 ? max_vec : 2;
  if (noise) max_vec = max_vec < align_vec(noise, 4) ? max_vec : align_vec(noise, 4);
  const int pa = (int)(reinterpret_cast<uintptr_t>(packed) & 3);
  if (pa != 0) max_vec = (pa == 2 && max_vec >= 2) ? 2 : 1;
  TileShape s;
  if (!choose_shape(D, max_vec, &s))
    return fail(EXB_ERR_UNSUPPORTED, "pack: D=%lld is beyond the register-tiled kernels (max 4096 when D%%4==0, 2048 when D%%2==0, 1024 otherwise)", D);
  p.tpt = s.tpt;
  if (dtype == kDtypeHalf) return launch_pack_bits<HalfBits>(p, bits, s, st);
  if (dtype == EXACT_DTYPE_F32) return launch_pack_bits<float>(p, bits, s, st);
  return launch_pack_bits<uint16_t>(p, bits, s, st);
}

int quantize_pack_half(const void* x, long long N, long long D, int bits, const float* noise, unsigned long long seed,
                       unsigned long long offset, long long row_offset, uint8_t* packed, uint16_t* scale, uint16_t* mn,
                       cudaStream_t st) {
  return pack_common(x, kDtypeHalf, N, D, D, bits, noise, nullptr, nullptr, seed, offset, row_offset, packed, scale, mn, nullptr,
                     nullptr, st);
}

template <int BITS, int STATS>
static int launch_unpack(const UnpackParams& p, const TileShape& s, cudaStream_t st) {
  const long long tiles = (p.N + 7) / 8;
  const int tiles_per_cta = s.block / s.tpt;
  const long long ctas = (tiles + tiles_per_cta - 1) / tiles_per_cta;
  int grid = 1;
#define EXB_UNPACK_CASE(VEC_, V_)                                                      \
  if (s.vec == VEC_ && s.v == V_) {                                                    \
    auto k = unpack_dequant_kernel<BITS, VEC_, V_, STATS>;                                \
    int rc = persistent_grid(k, s.block, ctas, &grid);                                 \
    if (rc) return rc;                                                                 \
    k<<<grid, s.block, 0, st>>>(p);                                                    \
    EXB_CUDA_OK(cudaGetLastError());                                                   \
    return EXB_OK;                                                                     \
  }
  EXB_UNPACK_CASE(4, 1) EXB_UNPACK_CASE(4, 2) EXB_UNPACK_CASE(4, 4)
  EXB_UNPACK_CASE(2, 1) EXB_UNPACK_CASE(2, 2) EXB_UNPACK_CASE(2, 4)
  EXB_UNPACK_CASE(1, 1) EXB_UNPACK_CASE(1, 2) EXB_UNPACK_CASE(1, 4)
#undef EXB_UNPACK_CASE
  return fail(EXB_ERR_UNSUPPORTED, "no unpack kernel for vec=%d v=%d", s.vec, s.v);
}

// stats: the STATS of the kernel
static int unpack_common(const uint8_t* packed, int bits, const void* scale, const void* min, int stats, long long N, long long D,
                         void* out, cudaStream_t st) {
  EXB_REQUIRE(bits == 1 || bits == 2 || bits == 4 || bits == 8, "bits must be 1, 2, 4 or 8 (got %d)", bits);
  EXB_REQUIRE(N >= 0 && D >= 0, "unpack: negative shape");
  if (N == 0 || D == 0) return EXB_OK;
  EXB_REQUIRE(packed && scale && min && out, "unpack: null pointer");
  int max_vec = align_vec(out, stats == 2 ? 2 : 4);
  if (D % 2 != 0 && max_vec == 4 && D < (1LL << 31)) {
    UnpackParams p{};
    p.packed = packed; p.scale = scale; p.mn = min; p.out = out; p.N = N; p.D = D;
    long long blocks = (N * D + 1023) / 1024;
    if (blocks > (long long)sm_count() * 16) blocks = (long long)sm_count() * 16;
#define EXB_FLAT(BITS_)                                                                                        \
  if (stats == 2) unpack_flat_kernel<BITS_, 2><<<(int)blocks, 256, 0, st>>>(p);                                \
  else if (stats == 1) unpack_flat_kernel<BITS_, 1><<<(int)blocks, 256, 0, st>>>(p);                           \
  else unpack_flat_kernel<BITS_, 0><<<(int)blocks, 256, 0, st>>>(p);                                           \
  break
    switch (bits) {
      case 1: EXB_FLAT(1);
      case 2: EXB_FLAT(2);
      case 4: EXB_FLAT(4);
      default: EXB_FLAT(8);
    }
#undef EXB_FLAT
    EXB_CUDA_OK(cudaGetLastError());
    return EXB_OK;
  }
  const int pa = (int)(reinterpret_cast<uintptr_t>(packed) & 3);
  if (pa != 0) max_vec = (pa == 2 && max_vec >= 2) ? 2 : 1;
  TileShape s;
  if (!choose_shape(D, max_vec, &s))
    return fail(EXB_ERR_UNSUPPORTED, "unpack: D=%lld is beyond the register-tiled kernels", D);
  UnpackParams p;
  p.packed = packed; p.scale = scale; p.mn = min; p.out = out; p.N = N; p.D = D; p.tpt = s.tpt;
  p.vec_stats = (reinterpret_cast<uintptr_t>(scale) % 16 == 0 && reinterpret_cast<uintptr_t>(min) % 16 == 0) ? 1 : 0;
#define EXB_UNPACK_STATS(BITS_)                                                                             \
  return stats == 2 ? launch_unpack<BITS_, 2>(p, s, st) : stats == 1 ? launch_unpack<BITS_, 1>(p, s, st)    \
                                                                     : launch_unpack<BITS_, 0>(p, s, st)
  switch (bits) {
    case 1: EXB_UNPACK_STATS(1);
    case 2: EXB_UNPACK_STATS(2);
    case 4: EXB_UNPACK_STATS(4);
    default: EXB_UNPACK_STATS(8);
  }
#undef EXB_UNPACK_STATS
}

int unpack_half(const uint8_t* packed, int bits, const void* scale, const void* min, long long N, long long D, void* out,
                cudaStream_t st) {
  return unpack_common(packed, bits, scale, min, 2, N, D, out, st);
}

}  // namespace exb

using namespace exb;

extern "C" {

int exact_quantize_pack(const void* x, int dtype, int64_t N, int64_t D, int bits, const float* noise,
                        uint64_t seed, uint64_t offset, int64_t row_offset, uint8_t* packed,
                        uint16_t* scale_bf16, uint16_t* min_bf16, float* scale_f32, float* min_f32,
                        void* stream) {
  return pack_common(x, dtype, N, D, D, bits, noise, nullptr, nullptr, seed, offset, row_offset, packed,
                     scale_bf16, min_bf16, scale_f32, min_f32, (cudaStream_t)stream);
}

int exact_quantize_pack_rows(const void* x, int dtype, int64_t N, int64_t D, int64_t ldx, int bits, uint64_t seed, uint64_t offset,
                             int64_t row_offset, uint8_t* packed, uint16_t* scale_bf16, uint16_t* min_bf16, void* stream) {
  EXB_REQUIRE(ldx >= D && ldx < (1LL << 28), "quantize_pack_rows: the pitch must be at least the row and below 2^28");
  return pack_common(x, dtype, N, D, ldx, bits, nullptr, nullptr, nullptr, seed, offset, row_offset, packed, scale_bf16, min_bf16,
                     nullptr, nullptr, (cudaStream_t)stream);
}

int exact_pack_single_precision(const void* data, int dtype, const float* min, const float* scale,
                                int64_t N, int64_t D, int bits, const float* noise, uint64_t seed,
                                uint64_t offset, int64_t row_offset, uint8_t* packed, void* stream) {
  if (N > 0 && D > 0) EXB_REQUIRE(min != nullptr && scale != nullptr, "pack_single_precision: null min/scale");
  return pack_common(data, dtype, N, D, D, bits, noise, min, scale, seed, offset, row_offset, packed,
                     nullptr, nullptr, nullptr, nullptr, (cudaStream_t)stream);
}

int exact_unpack_single_precision(const uint8_t* packed, int bits, const void* scale, const void* min,
                                  int stats_dtype, int64_t N, int64_t D, float* out, void* stream) {
  EXB_REQUIRE(stats_dtype == EXACT_DTYPE_F32 || stats_dtype == EXACT_DTYPE_BF16,
              "unpack: scale/min dtype must be EXACT_DTYPE_F32 or EXACT_DTYPE_BF16 (got %d)", stats_dtype);
  return unpack_common(packed, bits, scale, min, stats_dtype == EXACT_DTYPE_BF16 ? 1 : 0, N, D, out, (cudaStream_t)stream);
}

}  // extern "C"

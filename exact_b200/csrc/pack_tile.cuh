// Quantise + pack of tiles held in registers: the kernels, compiled for one input type each by pack_f32.cu, pack_bf16.cu and
// pack_half.cu (chosen and launched by pack.cu).
#pragma once
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

// Four adjacent elements of a row as loaded, whatever the width of the rows allows for an access: with chunks of two columns or
// one, a chunk's share of the addresses, of the byte assembly and (odd columns) of a noise block drawn for one column of two made
// narrow accesses cost 26 instructions an element against 15 to 18 (80 M elements, INT2, us, before and now: 17 columns fp32 334
// and 188, 47 182 and 137, 101 176 and 109, 601 135 and 103, 1,023 127 and 87; bf16 322 and 180, 183 and 128, 177 and 114, 160 and
// 98, 185 and 80).
// The elements are kept as loaded; 16-bit types stay packed in pairs: half the registers of the widened tile, and
// their minimum and maximum are taken two at a time.  ACC: elements per access (4, 2 or 1, what the rows' alignment allows; 0: one
// element too, of 16-bit rows that are pitched or start off a pair, see load_unaligned_tile);
// `have` of the four exist (always 4 with ACC == 4); the others repeat the first, by the address: with
// a predicate on each access the loads of a tile waited for one another (30 columns 204 us, 47 columns 248).
template <typename InT>
struct Raw {
  uint32_t w[2];
  template <int ACC>
  __device__ __forceinline__ void load(const InT* p, int have) {
    if (ACC == 4) {
      const uint2 t = __ldcs(reinterpret_cast<const uint2*>(p));
      w[0] = t.x;
      w[1] = t.y;
    } else if (ACC == 2) {
      w[0] = __ldcs(reinterpret_cast<const uint32_t*>(p));
      w[1] = __ldcs(reinterpret_cast<const uint32_t*>(p + (have > 2 ? 2 : 0)));
    } else {
      const uint16_t* q = reinterpret_cast<const uint16_t*>(p);
      uint32_t e[4];
#pragma unroll
      for (int i = 0; i < 4; i++) e[i] = __ldcs(q + (have > i ? i : 0));
      w[0] = __byte_perm(e[0], e[1], 0x5410);
      w[1] = __byte_perm(e[2], e[3], 0x5410);
    }
  }
  // Row r of a full tile with an odd number of columns whose first element lies on a pair: whole pairs are loaded, which start at
  // the element in front in odd rows.  The pairs that are read lie inside the tile: an odd row is not its first, an even one not
  // its last.
  static __device__ __forceinline__ void load_pairs(const InT* p, int r, int have, uint32_t (&m)[3]) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (r & 1));
    m[0] = __ldcs(q);
    m[1] = __ldcs(q + (have > 1 ? 1 : 0));
    if (r & 1) m[2] = __ldcs(q + (have > 3 ? 2 : have > 1 ? 1 : 0));
  }
  __device__ __forceinline__ void from_pairs(const uint32_t (&m)[3], int r, int have) {
    if (r & 1) {
      const uint32_t sel = have > 1 ? 0x5432u : 0x3232u;
      w[0] = __byte_perm(m[0], m[1], sel);
      w[1] = __byte_perm(m[1], m[2], sel);
    } else {
      w[0] = __byte_perm(m[0], 0u, have > 1 ? 0x3210u : 0x1010u);
      w[1] = __byte_perm(m[1], 0u, have > 3 ? 0x3210u : 0x1010u);
    }
  }
  // The four elements at p, which need not start on a pair (odd: they start on the second half of one), from the pairs they lie in.
  static __device__ __forceinline__ void load_around(const InT* p, int odd, int have, uint32_t (&m)[3]) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - odd);
    const int last = (odd + (have > 0 ? have < 4 ? have : 4 : 1) - 1) >> 1;   // the pair of the last one that exists
    m[0] = __ldcs(q);
    m[1] = __ldcs(q + (last > 0 ? 1 : 0));
    m[2] = __ldcs(q + last);
  }
  __device__ __forceinline__ void from_around(const uint32_t (&m)[3], int odd, int have) {
    const uint32_t first = have == 1 ? 0x1010u : 0x3210u, second = have & 1 && have < 4 ? 0x1010u : 0x3210u;
    const uint32_t first_odd = have == 1 ? 0x3232u : 0x5432u, second_odd = have >= 4 ? 0x5432u : have == 2 ? 0x1010u : 0x3232u;
    w[0] = __byte_perm(m[0], m[1], odd ? first_odd : first);
    w[1] = __byte_perm(m[1], m[2], odd ? second_odd : second);
  }
  __device__ __forceinline__ void clear() { w[0] = w[1] = 0u; }
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
    const uint32_t a = pair_min(w[0], w[1]), b = pair_max(w[0], w[1]);
    lo = min_nan3(lo, low(a), high(a));
    hi = max_nan3(hi, low(b), high(b));
  }
};
template <>
struct Raw<float> {
  float v[4];
  template <int ACC>
  __device__ __forceinline__ void load(const float* p, int have) {
    if (ACC == 4) {
      Ld<float, 4>::load(p, v);
    } else if (ACC == 2) {
      const float2 a = __ldcs(reinterpret_cast<const float2*>(p));
      const float2 b = __ldcs(reinterpret_cast<const float2*>(p + (have > 2 ? 2 : 0)));
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) v[i] = __ldcs(p + (have > i ? i : 0));
    }
  }
  __device__ __forceinline__ void clear() { v[0] = v[1] = v[2] = v[3] = 0.f; }
  __device__ __forceinline__ float at(int e) const { return v[e]; }
  __device__ __forceinline__ void range(float& lo, float& hi) const {
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      lo = min_nan3(lo, v[e], v[e + 1]);
      hi = max_nan3(hi, v[e], v[e + 1]);
    }
  }
};

// FULL: all 8 rows of the tile exist; one 64-bit base per chunk, rows addressed by 32-bit offsets.  have[v]: existing columns of
// chunk v (0: none).
template <typename InT, int ACC, int V, bool FULL>
__device__ __forceinline__ void load_tile(const InT* __restrict__ x, const TileCtx& c, long long tile,
                                          const long long (&col)[V], const int (&have)[V], Raw<InT> (&xv)[8][V]) {
  const long long row0 = tile << 3;
  const int rows_valid = FULL ? 8 : c.N - row0 >= 8 ? 8 : c.N > row0 ? (int)(c.N - row0) : 0;
  const unsigned Du = (unsigned)c.ldx;
#pragma unroll
  for (int v = 0; v < V; v++) {
    const InT* __restrict__ base = x + row0 * c.ldx + col[v];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      if ((FULL || r < rows_valid) && have[v] > 0) xv[r][v].template load<ACC>(base + r * Du, have[v]);
      else xv[r][v].clear();
    }
  }
}
// The same of a full tile with an odd number of 16-bit columns: all loads, then what belongs to a row.
template <typename InT, int V>
__device__ __forceinline__ void load_odd_tile(const InT* __restrict__ x, const TileCtx& c, long long tile,
                                              const long long (&col)[V], const int (&have)[V], Raw<InT> (&xv)[8][V]) {
#pragma unroll
  for (int v = 0; v < V; v++) {
    const InT* __restrict__ base = x + (tile << 3) * c.ldx + (have[v] > 0 ? col[v] : 0);
    uint32_t m[8][3];
#pragma unroll
    for (int r = 0; r < 8; r++) Raw<InT>::load_pairs(base + r * (unsigned)c.ldx, r, have[v], m[r]);
#pragma unroll
    for (int r = 0; r < 8; r++) xv[r][v].from_pairs(m[r], r, have[v]);
  }
}
// The same of 16-bit rows that start anywhere (of any pitch and base).  The pairs that hold a row's ends may reach one element past
// either of them, so the tile has a row in front of it and one behind.
template <typename InT, int V>
__device__ __forceinline__ void load_unaligned_tile(const InT* __restrict__ x, const TileCtx& c, long long tile,
                                                    const long long (&col)[V], const int (&have)[V], Raw<InT> (&xv)[8][V]) {
  const int base_odd = (int)(reinterpret_cast<uintptr_t>(x) >> 1) & 1, pitch_odd = (int)(c.ldx & 1);
#pragma unroll
  for (int v = 0; v < V; v++) {
    const InT* __restrict__ base = x + (tile << 3) * c.ldx + (have[v] > 0 ? col[v] : 0);
    uint32_t m[8][3];
#pragma unroll
    for (int r = 0; r < 8; r++) Raw<InT>::load_around(base + r * (unsigned)c.ldx, (base_odd + r * pitch_odd) & 1, have[v], m[r]);
#pragma unroll
    for (int r = 0; r < 8; r++) xv[r][v].from_around(m[r], (base_odd + r * pitch_odd) & 1, have[v]);
  }
}

// The first `have` bytes of a word.
template <int ACC>
__device__ __forceinline__ void store_codes(uint8_t* p, uint32_t w, int have) {
  if (ACC == 4) {
    __stcs(reinterpret_cast<uint32_t*>(p), w);
  } else if (ACC == 2) {
    __stcs(reinterpret_cast<uint16_t*>(p), (uint16_t)w);
    if (have > 2) __stcs(reinterpret_cast<uint16_t*>(p) + 1, (uint16_t)(w >> 16));
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (have > i) __stcs(p + i, (uint8_t)(w >> 8 * i));
  }
}

// Four 8-bit codes -> one word with a code per byte.
__device__ __forceinline__ uint32_t bytes_of(const uint32_t (&code)[4]) {
  return __byte_perm(__byte_perm(code[0], code[1], 0x0040), __byte_perm(code[2], code[3], 0x0040), 0x5410);
}

__device__ __forceinline__ float round_to_half(float f) { return __half2float(__float2half_rn(f)); }
// half(half(x - min) * scale) of elements e and e + 1, widened: the paired half instructions round each result once, which is
// what rounding the fp32 difference and product of halves to half gives (24 >= 2 * 11 + 2 digits).
template <typename InT>
__device__ __forceinline__ f32x2 half_scaled(const Raw<InT>& x, int e, float mn, float sc) {
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

// Quantise the 8 x 4V register tile with stochastic rounding and assemble the packed bytes.
// MAGIC (only with FAST, and only when every scale of the tile is a finite non-zero number): the
// rounding is done by adding 1.5 * 2^23, the code being the low byte of the sum.
template <typename InT, int BITS, int ACC, int V, bool FAST, bool MAGIC>
__device__ __forceinline__ void quantize_rows(const PackParams& p, const TileCtx& c, long long tile, int rows_valid,
                                              const long long (&col)[V], const int (&have)[V],
                                              const Raw<InT> (&xv)[8][V], const float (&mn)[8], const float (&sc)[8]) {
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
    if (have[v] <= 0) continue;
    uint32_t acc[GPT];
#pragma unroll
    for (int g = 0; g < GPT; g++) acc[g] = 0u;
    // MAGIC and fp32 arithmetic: with Philox noise (at most 1 - 2^-9) no code exceeds 2^bits - 1, so the rows of a byte may be
    // added instead of masked and OR-ed, on the floats' bit patterns (the exponent's share of the sum lies above the low
    // byte): one multiply-add per element instead of 1.25 permutes, shifts and masks.
    constexpr bool SUM = MAGIC && !HALF;
    uint32_t sum[4];

    // One Philox block per 8-row tile and PAIR of columns: its 16 bytes are the noise of rows 0..7 of the
    // even and the odd column (byte 2 r + (column & 1)), 8 bits per element: u = (h + 0.5) / 256.
    constexpr int NP = 2;
    uint32_t w[NP][4];
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
        float un[4];
        if (!FAST && nbase != nullptr) {
          Raw<float> t;
          t.template load<ACC>(nbase + r * Du, have[v]);
#pragma unroll
          for (int e = 0; e < 4; e++) un[e] = t.v[e];
        }
        uint32_t code[4];
        const f32x2 mn2 = f2_pack(mn[r], mn[r]);
        const f32x2 sc2 = f2_pack(sc[r], sc[r]);
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          f32x2 u2;
          if (!FAST && nbase != nullptr) {
            u2 = f2_pack(un[e], un[e + 1]);
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
            const f32x2 a2 = f2_sub(f2_pack(xv[r][v].at(e), xv[r][v].at(e + 1)), mn2);
            t2 = f2_add(f2_fma(a2, sc2, u2), neg_half);
          }
          float t0, t1;
          if (MAGIC) {
            t2 = f2_add(t2, magic);
            f2_unpack(t2, t0, t1);
            code[e] = __float_as_uint(t0);            // low byte = rint(t); higher bytes are dropped below
            code[e + 1] = __float_as_uint(t1);
          } else {
            f2_unpack(t2, t0, t1);
            code[e] = __float2uint_rn(t0);
            code[e + 1] = __float2uint_rn(t1);
          }
        }
        if (SUM) {
#pragma unroll
          for (int e = 0; e < 4; e++)
            sum[e] = r % WPT == 0 ? code[e] : sum[e] + code[e] * (1u << ((r % WPT) * BITS));
          if (r % WPT == WPT - 1) acc[r / WPT] = bytes_of(sum);
          continue;
        }
        const uint32_t word = bytes_of(code);
        constexpr uint32_t kOnes = 0x01010101u;
        const int sh = (r % WPT) * BITS;
        if (sh == 0) acc[r / WPT] = word;
        else acc[r / WPT] |= (word << sh) & (kOnes * ((0xffu << sh) & 0xffu));  // uint8 narrowing per byte
      }
    }

    uint8_t* __restrict__ obase = p.packed + (tile * GPT) * c.D + col[v];
#pragma unroll
    for (int g = 0; g < GPT; g++) {
      if (FAST || tile * GPT + g < c.G) store_codes<ACC>(obase + g * Du, acc[g], have[v]);
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
//   two warps a tile (385 - 512 columns; fewer tiles than one-warp tiles want, from 257): 128 registers keep a fourth CTA of 128
//     threads resident.  320 columns, INT2: fp32 102 | 94, bf16 111 | 98, fp16 105 | 95;
//   several warps a tile, accesses of two elements or one: 601 columns, INT2: fp32 169 | 102, bf16 215 | 98.  With accesses of four
//     one stays the better bound (640 columns, INT8: fp32 85 | 84, fp16 82 | 93);
//   one warp a tile, two chunks, bf16 (132 - 256 columns): 200 columns, INT2 90 | 86 (fp32 78 | 80, left at one).
template <typename InT>
constexpr int resident_ctas(int acc, int v, int kind) {
  if (v != 2) return 1;
  if (acc < 4 && kind >= TILE_MULTI) return 2;
  return kind == TILE_PAIR || (kind == TILE_WARP && std::is_same<InT, uint16_t>::value) ? 2 : 1;
}

// FAST: the tile has all 8 rows and the noise is drawn from Philox.  Then there is no per-row
// validity test, and -- when all 8 scales are finite and non-zero, i.e. no row is constant or holds
// an infinity or a NaN -- round-to-nearest-even is done by adding 1.5 * 2^23 (the code is then the
// low byte of the float) instead of a float->int conversion.
template <typename InT, int BITS, int ACC, int V, int KIND, bool FAST>
__device__ __forceinline__ bool process_tile(const PackParams& p, const TileCtx& c, long long tile, int it,
                                             const long long (&col)[V], const int (&have)[V],
                                             const Raw<InT> (&xv)[8][V], float* s_part, float* s_fin) {
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
      if (have[v] > 0) xv[r][v].range(lo[r], hi[r]);
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
    quantize_rows<InT, BITS, ACC, V, true, true>(p, c, tile, 8, col, have, xv, mn, sc);
  } else {
    quantize_rows<InT, BITS, ACC, V, false, false>(p, c, tile, rows_valid, col, have, xv, mn, sc);
  }
  return true;
}

template <typename InT, int BITS, int ACC, int V, int KIND>
__global__ void __launch_bounds__(256, resident_ctas<InT>(ACC, V, KIND))
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
  int have[V];
#pragma unroll
  for (int v = 0; v < V; v++) {
    col[v] = (long long)(c.tl + v * c.tpt) * 4;
    have[v] = p.D - col[v] >= 4 ? 4 : (int)(p.D - col[v]);
  }

  // The next tile (one contiguous run of 8 * D elements) is pulled into L2 by a single bulk-prefetch
  // instruction while the current one is processed, so the register loads of the next iteration
  // find their lines on chip.
  const long long tile_bytes = 8 * p.D * (long long)sizeof(InT);
  const bool can_prefetch = p.ldx == p.D && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0 && (tile_bytes & 15) == 0;
  constexpr bool ODD16 = ACC == 1 && sizeof(InT) == 2, UNALIGNED16 = ACC == 0;   // ODD16: one run that starts on a pair
  const bool fast = p.noise == nullptr &&
                    (!ODD16 || ((p.ldx & 1) != 0 && p.ldx == p.D && (reinterpret_cast<uintptr_t>(p.x) & 3) == 0));
  Raw<InT> xv[8][V];
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
    // an unaligned tile's neighbours: none in front of the first, none certain behind the last
    if (fast && tile - in_warp + last_in_warp < (UNALIGNED16 ? num_tiles - 1 : full_tiles) && (!UNALIGNED16 || tile - in_warp > 0)) {
      if constexpr (UNALIGNED16) load_unaligned_tile<InT, V>(x, c, tile, col, have, xv);
      else if constexpr (ODD16) load_odd_tile<InT, V>(x, c, tile, col, have, xv);
      else load_tile<InT, ACC, V, true>(x, c, tile, col, have, xv);
      done = process_tile<InT, BITS, ACC, V, KIND, true>(p, c, tile, it, col, have, xv, s_part, s_fin);
      if (!done) ++it;  // the redo below exchanges its statistics through the other shared-memory buffer
    }
    if (!done) {
      load_tile<InT, ACC, V, false>(x, c, tile, col, have, xv);
      process_tile<InT, BITS, ACC, V, KIND, false>(p, c, tile, it, col, have, xv, s_part, s_fin);
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// Host side
struct TileShape {
  int vec, v, tpt, block;
};

template <auto KERNEL>
static int persistent_grid(int block, long long work_ctas) {
  const long long most = (long long)sm_count() * blocks_per_sm<KERNEL>(block);
  return (int)(work_ctas < 1 ? 1 : work_ctas < most ? work_ctas : most);
}

template <typename InT, int BITS>
static int launch_pack(const PackParams& p, const TileShape& s, cudaStream_t st) {
  const long long tiles = (p.N + 7) / 8;
  const int tiles_per_cta = s.block / s.tpt;
  const long long ctas = (tiles + tiles_per_cta - 1) / tiles_per_cta;
  const int kind = s.tpt < 32 ? TILE_SUB : s.tpt == 32 ? TILE_WARP : s.tpt == 64 ? TILE_PAIR : TILE_MULTI;
#define EXB_PACK_CASE(ACC_, V_, KIND_)                                                 \
  if (s.vec == ACC_ && s.v == V_ && kind == KIND_) {                                   \
    constexpr auto k = quantize_pack_kernel<InT, BITS, ACC_, V_, KIND_>;               \
    k<<<persistent_grid<k>(s.block, ctas), s.block, 0, st>>>(p);                       \
    EXB_CUDA_OK(cudaGetLastError());                                                   \
    return EXB_OK;                                                                     \
  }
#define EXB_PACK_CASES(ACC_)                                                                                    \
  EXB_PACK_CASE(ACC_, 1, TILE_SUB) EXB_PACK_CASE(ACC_, 1, TILE_WARP) EXB_PACK_CASE(ACC_, 2, TILE_WARP)          \
  EXB_PACK_CASE(ACC_, 3, TILE_WARP) EXB_PACK_CASE(ACC_, 2, TILE_PAIR) EXB_PACK_CASE(ACC_, 2, TILE_MULTI)
  EXB_PACK_CASES(4) EXB_PACK_CASES(2) EXB_PACK_CASES(1)
  EXB_PACK_CASE(4, 4, TILE_MULTI)
  if constexpr (sizeof(InT) == 2) {
    EXB_PACK_CASES(0)
    EXB_PACK_CASE(4, 5, TILE_WARP) EXB_PACK_CASE(2, 5, TILE_WARP)
  }
#undef EXB_PACK_CASES
#undef EXB_PACK_CASE
  return fail(EXB_ERR_UNSUPPORTED, "no pack kernel for vec=%d v=%d", s.vec, s.v);
}

template <typename InT>
int launch_pack_bits(const PackParams& p, int bits, const TileShape& s, cudaStream_t st) {
  switch (bits) {
    case 1: return launch_pack<InT, 1>(p, s, st);
    case 2: return launch_pack<InT, 2>(p, s, st);
    case 4: return launch_pack<InT, 4>(p, s, st);
    case 8: return launch_pack<InT, 8>(p, s, st);
  }
  return fail(EXB_ERR_ARG, "bits must be 1, 2, 4 or 8 (got %d)", bits);
}

}  // namespace exb

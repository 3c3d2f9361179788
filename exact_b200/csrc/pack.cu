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
// width.  `tpt` threads own one tile; each thread keeps 8 rows x V chunks x 4 columns in registers,
// so bytes are assembled thread-locally and stored up to four at a time, and the activation is read from
// HBM exactly once.  Row min/max go through redux.sync (folded shuffles when tpt < 32) and, when a
// tile spans several warps, a double-buffered shared-memory exchange with named barriers.  While a
// tile is processed, the next one (a contiguous run of 8*D elements) is pulled into L2 with one
// cp.async.bulk.prefetch.  The arithmetic uses the paired fp32 instructions of sm_100 (two elements per issue slot,
// each rounded exactly like the scalar instruction).
#include "pack_tile.cuh"

namespace exb {

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
__device__ __forceinline__ uint32_t load_bytes(const uint8_t* p) {
  if (VEC == 4) return __ldcs(reinterpret_cast<const uint32_t*>(p));
  if (VEC == 2) return __ldcs(reinterpret_cast<const uint16_t*>(p));
  return __ldcs(p);
}

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
          using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type>;
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
            using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type>;
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
        using Stat = Raw<typename std::conditional<HALF, HalfBits, uint16_t>::type>;
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

// The same for packing, whose chunks are four columns whatever the accesses: tiles of 8 rows x 4v columns per thread.  A one-warp
// tile of three chunks (257 - 384 columns), or of five in 16-bit types (513 - 640, 80 registers of data), leaves fewer lanes idle
// than several warps of two chunks, and none of them waits for another: 300 columns, 80 M elements, INT2, us: fp32 100 | 81, bf16
// 102 | 84, fp16 97 | 82; 516 columns bf16 102 | 90, fp16 96 | 88; 602 bf16 96 | 92, fp16 104 | 94; four chunks (400, 512 columns)
// and five of single accesses (601: bf16 98 | 108) lose.  It wants enough tiles for every SM, else more warps finish earlier.
static bool choose_pack_shape(long long N, long long D, int acc, bool wide, TileShape* s) {
  if (D > (acc == 4 ? 4096 : acc == 2 ? 2048 : 1024)) return false;
  const int C = (int)((D + 3) / 4), v = (C + 31) / 32;
  if (C <= 32) {
    s->v = 1;
    s->tpt = pow2ceil(C) < 8 ? 8 : pow2ceil(C);
  } else if (v == 2 || ((v == 3 || (v == 5 && !wide && acc > 1)) && (N + 7) / 8 >= 8LL * sm_count())) {
    s->v = v;
    s->tpt = 32;
  } else {
    s->v = C <= 512 ? 2 : 4;
    s->tpt = ((C + s->v - 1) / s->v + 31) / 32 * 32;
  }
  s->vec = acc;
  s->block = s->tpt >= 128 ? s->tpt : s->tpt * (128 / s->tpt);
  return true;
}

extern template int launch_pack_bits<float>(const PackParams&, int, const TileShape&, cudaStream_t);
extern template int launch_pack_bits<uint16_t>(const PackParams&, int, const TileShape&, cudaStream_t);
extern template int launch_pack_bits<HalfBits>(const PackParams&, int, const TileShape&, cudaStream_t);

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
  if (!choose_pack_shape(N, D, D % 4 == 0 ? max_vec : D % 2 == 0 && max_vec >= 2 ? 2 : 1, dtype == EXACT_DTYPE_F32, &s))
    return fail(EXB_ERR_UNSUPPORTED, "pack: D=%lld is beyond the register-tiled kernels (max 4096 when D%%4==0, 2048 when D%%2==0, 1024 otherwise)", D);
  p.tpt = s.tpt;
  // Single accesses of 16-bit rows: a run of odd rows that starts on a pair is read in pairs whose halves are known (ACC 1); rows
  // that are pitched or start elsewhere in pairs too, whose halves depend on pitch and base (ACC 0).  80 M elements of bf16, INT2,
  // us, element by element | so: 101 columns in rows of 104 321 | 118, 301 of 305 471 | 109, 600 of 605 265 | 101; the run's form
  // takes 109 for 101 columns of 101, one form for both 111 and, at 47 columns, 158 instead of 123 (registers).
  if (s.vec == 1 && eb == 2 && noise == nullptr &&
      ((ldx & 1) == 0 || ldx != D || (reinterpret_cast<uintptr_t>(x) & 3) != 0))
    s.vec = 0;
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
#define EXB_UNPACK_CASE(VEC_, V_)                                                      \
  if (s.vec == VEC_ && s.v == V_) {                                                    \
    constexpr auto k = unpack_dequant_kernel<BITS, VEC_, V_, STATS>;                   \
    k<<<persistent_grid<k>(s.block, ctas), s.block, 0, st>>>(p);                       \
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

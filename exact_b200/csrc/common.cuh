// Shared device helpers of the exact_b200 CUDA library (sm_100a only).
#pragma once
#include <atomic>
#include <cmath>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "exact_b200 kernels are written for sm_100a (B200) only"
#endif

namespace exb {

// ---- host-side error plumbing -------------------------------------------------------------------
enum Status : int {
  EXB_OK = 0,
  EXB_ERR_ARG = 1,       // bad argument (null pointer, unsupported bits / dtype / size, misalignment)
  EXB_ERR_CUDA = 2,      // a CUDA runtime call failed; see exact_last_error()
  EXB_ERR_UNSUPPORTED = 3,
  EXB_ERR_DEVICE = 4,    // a kernel reported a device-side status (bounded wait expired)
};

char* last_error_buf();  // thread-local, defined in capi.cu

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buf(), 512, fmt, ap);
  va_end(ap);
  return code;
}

#define EXB_CUDA_OK(expr)                                                                     \
  do {                                                                                        \
    cudaError_t _e = (expr);                                                                  \
    if (_e != cudaSuccess)                                                                    \
      return ::exb::fail(::exb::EXB_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,                 \
                         cudaGetErrorString(_e), __FILE__, __LINE__);                         \
  } while (0)

#define EXB_REQUIRE(cond, ...)                                                                \
  do {                                                                                        \
    if (!(cond)) return ::exb::fail(::exb::EXB_ERR_ARG, __VA_ARGS__);                         \
  } while (0)

int sm_count();  // cached multiProcessorCount of the current device (capi.cu)

// Device address of the library-wide status word of the current device (capi.cu), or null without a device.
// Kernels with bounded on-chip waits OR one of these codes into it when a wait expires; exact_status() reads it.
// The word lives in page-locked host memory: the host looks at it without a copy or an event behind the launches.
int* status_word_ptr();
enum DeviceStatusBits : int { EXB_STATUS_RP_PACK = 1, EXB_STATUS_UNPACK_RP = 2, EXB_STATUS_LINEAR = 4, EXB_STATUS_GRAD_WEIGHT = 8 };

// Round keys of Philox4x32-10 for a 64-bit seed; lives in kernel parameters (constant bank) so the
// per-round key XOR needs no register.
struct PhiloxKey {
  uint32_t rk[20];
};
inline PhiloxKey make_philox_key(uint64_t seed) {
  PhiloxKey k;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; r++) {
    k.rk[2 * r] = k0;
    k.rk[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return k;
}

#ifdef __CUDACC__
// Blocks of a kernel without dynamic shared memory that fit on an SM of the current device, at least one.  A property of the
// compiled kernel, so the latest answer is kept per kernel, with its device and block size in the same word, which any thread may
// replace.
template <auto KERNEL>
inline int blocks_per_sm(int threads) {
  static std::atomic<uint64_t> latest{0};
  int dev = 0, blocks = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  const uint64_t key = (uint64_t)(uint32_t)(dev + 1) << 32 | (uint64_t)(uint32_t)threads << 16;
  const uint64_t kept = latest.load(std::memory_order_relaxed);
  if ((kept & ~(uint64_t)0xffff) == key) return (int)(kept & 0xffff);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, KERNEL, threads, 0) != cudaSuccess || blocks < 1) return 1;
  latest.store(key | (uint64_t)blocks, std::memory_order_relaxed);
  return blocks;
}
// Blocks of a kernel whose blocks walk over the data: as many as are resident at once, or fewer when there is less to do.  With
// more, the last round of blocks leaves SMs idle (at 40 registers six blocks of 256 threads fit; eight per SM took two rounds, the
// second a third full).
template <auto KERNEL>
inline int resident_blocks(int threads, long long want) {
  int per_sm = blocks_per_sm<KERNEL>(threads);
  if (per_sm > 8) per_sm = 8;      // what the workspaces of partial sums are sized for
  const long long most = (long long)sm_count() * per_sm;
  return (int)(want < 1 ? 1 : want < most ? want : most);
}
#endif

// What dropout multiplies kept values by, and divides their gradients by.
struct DropoutScale {
  float pinv;            // float(1 / (1 - p)), quantization_cuda_kernel.cu:455
  float p1m;             // float(1 - p), quantization.cc:120
  float p1m_inv_exact;   // 1 / p1m when p1m is a power of two (then g / p1m == g * that, bit for bit), else 0
};
inline DropoutScale dropout_scale(float prob) {
  DropoutScale s;
  s.pinv = (float)(1.0 / (1.0 - (double)prob));
  s.p1m = (float)(1.0 - (double)prob);
  int ex = 0;
  const float mant = frexpf(s.p1m, &ex);   // p1m = mant * 2^ex, mant in [0.5, 1)
  s.p1m_inv_exact = (s.p1m > 0.f && mant == 0.5f && ex > -120 && ex < 120) ? ldexpf(1.f, 1 - ex) : 0.f;
  return s;
}

#ifdef __CUDACC__
// A kept gradient: g / float(1 - p) (quantization_cuda_kernel.cu:565-569); a power-of-two divisor (p = 0.5, 0.75, ...) is an exact
// scaling, done as one multiply.
__device__ __forceinline__ float dropout_grad(float g, float p1m, float p1m_inv_exact) {
  return p1m_inv_exact != 0.f ? __fmul_rn(g, p1m_inv_exact) : __fdiv_rn(g, p1m);
}
// 16-bit draw -> (h + 0.5) / 65536, exact.
__device__ __forceinline__ float dropout_uniform(uint32_t h) { return __fmaf_rn((float)h, 1.52587890625e-05f, 7.62939453125e-06f); }

// CTAs and kernels that give up at the same moment all leave their bit: an atomic on mapped host memory is one for all threads of
// the device that maps it, and the host writes the word only to clear or set it, after the stream it was asked for.
__device__ __forceinline__ void raise_status(int* word, int bit) {
  if (word == nullptr) return;
  atomicOr(word, bit);
  __threadfence_system();
}

// ---- device helpers -----------------------------------------------------------------------------

// Philox4x32-10 (Salmon et al., SC'11).  Counter (c0..c3), round keys from the constant bank.
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                              const PhiloxKey& key, uint32_t (&out)[4]) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c0;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ key.rk[2 * r];
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ key.rk[2 * r + 1];
    c1 = (uint32_t)p1;
    c3 = (uint32_t)p0;
    c0 = n0;
    c2 = n2;
  }
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
}

// 16-bit field h -> (h + 0.5) * 2^-16 in (0,1), without an int->float conversion:
// 0x3F800000 | (h << 7) is 1 + h*2^-16; subtracting (1 - 2^-17) is exact.
__device__ __forceinline__ float u16_lo_to_unit(uint32_t w) {
  return __uint_as_float(((w << 7) & 0x007fff80u) | 0x3f800000u) - 0.99999237060546875f;
}
__device__ __forceinline__ float u16_hi_to_unit(uint32_t w) {
  return __uint_as_float(((w >> 9) & 0x007fff80u) | 0x3f800000u) - 0.99999237060546875f;
}
// 32-bit draw r -> r * 2^-32 + 2^-33 in (0,1] (the usual "uniform excluding zero" map).
__device__ __forceinline__ float u32_to_unit(uint32_t r) {
  return __fmaf_rn((float)r, 2.3283064365386963e-10f, 1.1641532182693481e-10f);
}

// Two fp32 lanes in one 64-bit register and the paired arithmetic of sm_100 (each lane rounds exactly
// like the scalar instruction).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// 16-bit field of a Philox word -> the float 1 + h * 2^-23 (bits 0x3F80:h), by one byte permute.
// noise16_to_unit() turns a pair of those into (h + 0.5) * 2^-16 with one paired FMA:
// (1 + h 2^-23) * 128 - (128 - 2^-17), exact.
__device__ __forceinline__ float u16_lo_to_1p(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7610)); }
__device__ __forceinline__ float u16_hi_to_1p(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7632)); }
__device__ __forceinline__ f32x2 noise16_to_unit(f32x2 one_plus) {
  return f2_fma(one_plus, f2_pack(128.f, 128.f), f2_pack(-127.99999237060546875f, -127.99999237060546875f));
}

// Byte k (0..3, may be a run-time value) of a Philox word -> the float 1 + h * 2^-23 (bits 0x3F8000:h), by one
// byte permute; noise8_to_unit() turns those into (h + 0.5) * 2^-8 with one FMA:
// (1 + h 2^-23) * 2^15 - (2^15 - 2^-9), exact.
__device__ __forceinline__ float u8_to_1p(uint32_t w, uint32_t k) {
  return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7640u + k));
}
__device__ __forceinline__ f32x2 noise8_to_unit(f32x2 one_plus) {
  return f2_fma(one_plus, f2_pack(32768.f, 32768.f), f2_pack(-32767.998046875f, -32767.998046875f));
}
__device__ __forceinline__ float noise8_to_unit(float one_plus) {
  return __fmaf_rn(one_plus, 32768.f, -32767.998046875f);
}

// NaN-propagating min/max (torch.min / torch.max semantics) and their warp-wide forms.  redux.sync on
// f32 is an sm_100a instruction.
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float min_nan3(float a, float b, float c) {   // three operands: an sm_100 instruction
  float r;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max_nan3(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float redux_min_nan(float v, unsigned mask) {
  float r;
  asm volatile("redux.sync.min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "r"(mask));
  return r;
}
__device__ __forceinline__ float redux_max_nan(float v, unsigned mask) {
  float r;
  asm volatile("redux.sync.max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "r"(mask));
  return r;
}

// Named barrier over `nthreads` threads (a multiple of 32) of the CTA.
template <int ID>
__device__ __forceinline__ void named_barrier(int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(nthreads) : "memory");
}

// fp32 -> bf16 bits, round to nearest even, NaN -> 0x7FC0 (what Tensor.to(torch.bfloat16) produces).
__device__ __forceinline__ uint16_t f32_to_bf16_bits(float f) {
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7fffffffu) > 0x7f800000u) return 0x7fc0;
  return (uint16_t)((u + 0x7fffu + ((u >> 16) & 1u)) >> 16);
}
__device__ __forceinline__ float bf16_bits_to_f32(uint16_t h) {
  return __uint_as_float(((uint32_t)h) << 16);
}

// Streaming (read-once / write-once) global accesses of 1, 2 or 4 elements.
template <typename T, int VEC>
struct Ld;
template <>
struct Ld<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[4]) {
    float4 v = __ldcs(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <>
struct Ld<float, 2> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[2]) {
    float2 v = __ldcs(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  }
};
template <>
struct Ld<float, 1> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[1]) { o[0] = __ldcs(p); }
};
// bf16 stored as uint16_t bits; widening to fp32 is exact.
template <>
struct Ld<uint16_t, 4> {
  static __device__ __forceinline__ void load(const uint16_t* p, float (&o)[4]) {
    uint2 v = __ldcs(reinterpret_cast<const uint2*>(p));
    o[0] = __uint_as_float(v.x << 16); o[1] = __uint_as_float(v.x & 0xffff0000u);
    o[2] = __uint_as_float(v.y << 16); o[3] = __uint_as_float(v.y & 0xffff0000u);
  }
};
template <>
struct Ld<uint16_t, 2> {
  static __device__ __forceinline__ void load(const uint16_t* p, float (&o)[2]) {
    uint32_t v = __ldcs(reinterpret_cast<const uint32_t*>(p));
    o[0] = __uint_as_float(v << 16); o[1] = __uint_as_float(v & 0xffff0000u);
  }
};
template <>
struct Ld<uint16_t, 1> {
  static __device__ __forceinline__ void load(const uint16_t* p, float (&o)[1]) {
    o[0] = __uint_as_float(((uint32_t)__ldcs(p)) << 16);
  }
};

template <int VEC>
struct StBytes;
template <>
struct StBytes<4> {
  static __device__ __forceinline__ void store(uint8_t* p, const uint32_t (&b)[4]) {
    __stcs(reinterpret_cast<uint32_t*>(p), b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24));
  }
  static __device__ __forceinline__ void load(const uint8_t* p, uint32_t (&b)[4]) {
    uint32_t w = __ldcs(reinterpret_cast<const uint32_t*>(p));
    b[0] = w & 0xff; b[1] = (w >> 8) & 0xff; b[2] = (w >> 16) & 0xff; b[3] = w >> 24;
  }
};
template <>
struct StBytes<2> {
  static __device__ __forceinline__ void store(uint8_t* p, const uint32_t (&b)[2]) {
    __stcs(reinterpret_cast<uint16_t*>(p), (uint16_t)(b[0] | (b[1] << 8)));
  }
  static __device__ __forceinline__ void load(const uint8_t* p, uint32_t (&b)[2]) {
    uint32_t w = __ldcs(reinterpret_cast<const uint16_t*>(p));
    b[0] = w & 0xff; b[1] = (w >> 8) & 0xff;
  }
};
template <>
struct StBytes<1> {
  static __device__ __forceinline__ void store(uint8_t* p, const uint32_t (&b)[1]) {
    __stcs(p, (uint8_t)b[0]);
  }
  static __device__ __forceinline__ void load(const uint8_t* p, uint32_t (&b)[1]) { b[0] = __ldcs(p); }
};

template <int VEC>
struct StF32;
template <>
struct StF32<4> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
  }
};
template <>
struct StF32<2> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[2]) {
    __stcs(reinterpret_cast<float2*>(p), make_float2(v[0], v[1]));
  }
};
template <>
struct StF32<1> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[1]) { __stcs(p, v[0]); }
};
#endif  // __CUDACC__

}  // namespace exb

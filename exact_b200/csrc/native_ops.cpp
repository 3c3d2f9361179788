// The ops of native.h: one function per entry point of the C ABI, with the checks and messages of the reference's
// extension modules (ext_common.h:2-32: CUDA, contiguous, rank, dtype).
#include "native.h"

#include <chrono>
#include <cuda_runtime_api.h>

namespace exb {

Library lib;
Accounting acct;

int64_t now_ns() {
  return std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
void timed_begin(const char* name, const CallInfo& info, cudaStream_t st, TimedCall& rec) {
  rec.name = name;
  rec.bytes = info.bytes;
  rec.l2_bytes = info.l2_bytes;
  rec.edge_columns = info.edge_columns;
  rec.flops = info.flops;
  cudaEventCreate(&rec.begin);
  cudaEventCreate(&rec.end);
  cudaEventRecord(rec.begin, st);
}
void timed_end(cudaStream_t st, TimedCall& rec) {
  cudaEventRecord(rec.end, st);
  std::lock_guard<std::mutex> lock(acct.mu);
  acct.calls.push_back(rec);
}
void library_failure(const char* name, int rc) {
  const char* msg = lib.exact_last_error();
  throw LibraryError(std::string(name) + " failed (code " + std::to_string(rc) + "): " + (msg ? msg : ""));
}

namespace {

void check_tensor(const Tensor& t, const char* name, int64_t dim) {
  if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor!");
  if (!t.is_contiguous()) throw std::runtime_error(std::string(name) + " must be contiguous!");
  if (dim >= 0 && t.dim() != dim) throw std::runtime_error("The dimension of " + std::string(name) + " is not correct!");
}
void check_type(bool ok, const char* name) {
  if (!ok) throw std::runtime_error("The type of " + std::string(name) + " is not correct!");
}
void same_device(const Tensor& a, const Tensor& b) {
  if (a.get_device() != b.get_device()) throw LibraryError("arguments live on different CUDA devices");
}
void same_device(const Tensor& a, const OptTensor& b) {
  if (b) same_device(a, *b);
}
void check_bits(int64_t bits) {
  if (bits != 1 && bits != 2 && bits != 4 && bits != 8) throw std::runtime_error("bits must be 1, 2, 4 or 8");
}
template <class T = void>
T* ptr(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <class T = void>
T* ptr(const OptTensor& t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

Tensor empty(at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
  return at::empty(shape, like.options().dtype(type).requires_grad(false));
}
int64_t elem(const Tensor& t) { return (int64_t)t.element_size(); }

}  // namespace

Packed quantize_pack(const Tensor& x, int64_t bits, const OptTensor& noise, uint64_t seed, uint64_t offset, int64_t row_offset) {
  check_tensor(x, "data", 2);
  const auto type = x.scalar_type();
  check_type(type == at::kFloat || type == at::kBFloat16 || type == at::kHalf, "data");
  check_bits(bits);
  const int64_t N = x.size(0), D = x.size(1);
  if (noise) {
    check_tensor(*noise, "noise", 2);
    check_type(noise->scalar_type() == at::kFloat, "noise");
    if (noise->size(0) != N || noise->size(1) != D) throw std::runtime_error("noise must have the shape of data");
    same_device(x, *noise);
    seed = offset = 0;
  }
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t bytes = lib.exact_packed_bytes(N, D, (int)bits);
  Packed q;
  q.codes = empty({bytes + 1}, at::kChar, x);
  const auto stat = type == at::kHalf ? at::kHalf : at::kBFloat16;   // ops.py:80-83
  q.scale = empty({N}, stat, x);
  q.mn = empty({N}, stat, x);
  if (type == at::kHalf) {
    invoke("exact_quantize_pack_f16", {2 * N * D * 2 + bytes + 4 * N}, [&](void* st) {
      return lib.exact_quantize_pack_f16(ptr<uint16_t>(x), N, D, (int)bits, ptr<float>(noise), seed, offset, row_offset,
                                         ptr<uint8_t>(q.codes), ptr<uint16_t>(q.scale), ptr<uint16_t>(q.mn), st);
    });
  } else {
    invoke("exact_quantize_pack", {N * D * elem(x) + bytes + 4 * N}, [&](void* st) {
      return lib.exact_quantize_pack(ptr(x), type == at::kFloat ? EXACT_DTYPE_F32 : EXACT_DTYPE_BF16, N, D, (int)bits,
                                     ptr<float>(noise), seed, offset, row_offset, ptr<uint8_t>(q.codes),
                                     ptr<uint16_t>(q.scale), ptr<uint16_t>(q.mn), nullptr, nullptr, st);
    });
  }
  return q;
}

Packed quantize_pack_rows(const Tensor& x, int64_t bits, uint64_t seed, uint64_t offset, int64_t row_offset) {
  check_type(x.is_cuda() && x.dim() == 2 && x.stride(1) == 1 && x.scalar_type() == at::kFloat, "data");
  check_bits(bits);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t N = x.size(0), D = x.size(1), bytes = lib.exact_packed_bytes(N, D, (int)bits);
  Packed q{empty({bytes + 1}, at::kChar, x), empty({N}, at::kBFloat16, x), empty({N}, at::kBFloat16, x)};
  invoke("exact_quantize_pack", {N * D * 4 + bytes + 4 * N}, [&](void* st) {
    return lib.exact_quantize_pack_rows(ptr(x), EXACT_DTYPE_F32, N, D, x.stride(0), (int)bits, seed, offset, row_offset,
                                        ptr<uint8_t>(q.codes), ptr<uint16_t>(q.scale), ptr<uint16_t>(q.mn), st);
  });
  return q;
}

Tensor unpack(const Tensor& codes, int64_t bits, const Tensor& scale, const Tensor& mn, int64_t N, int64_t D) {
  if (!codes.is_cuda() || !codes.is_contiguous() || codes.dim() != 1 || codes.scalar_type() != at::kChar)
    throw std::runtime_error("The type of data is not correct!");
  check_tensor(scale, "scale", 1);
  check_tensor(mn, "min", 1);
  const auto type = scale.scalar_type();
  check_type(type == at::kFloat || type == at::kBFloat16 || type == at::kHalf, "scale");
  if (mn.scalar_type() != type) throw std::runtime_error("scale and min must have the same dtype");
  check_bits(bits);
  same_device(codes, scale);
  same_device(codes, mn);
  const int64_t need = lib.exact_packed_bytes(N, D, (int)bits);
  if (codes.numel() < need || scale.numel() < N || mn.numel() < N)
    throw std::runtime_error("packed stream or statistics shorter than N x group_size requires");
  c10::cuda::CUDAGuard guard(codes.device());
  if (type == at::kHalf) {
    // the output has the statistics' dtype (quantization_cuda_kernel.cu:194-195): fp16, half arithmetic
    Tensor out = empty({N, D}, at::kHalf, codes);
    invoke("exact_unpack_single_precision_f16", {need + 4 * N + 2 * N * D}, [&](void* st) {
      return lib.exact_unpack_single_precision_f16(ptr<uint8_t>(codes), (int)bits, ptr<uint16_t>(scale), ptr<uint16_t>(mn), N, D,
                                                   ptr<uint16_t>(out), st);
    });
    return out;
  }
  Tensor out = empty({N, D}, at::kFloat, codes);
  invoke("exact_unpack_single_precision", {need + 2 * N * elem(scale) + 4 * N * D}, [&](void* st) {
    return lib.exact_unpack_single_precision(ptr<uint8_t>(codes), (int)bits, ptr(scale), ptr(mn),
                                             type == at::kFloat ? EXACT_DTYPE_F32 : EXACT_DTYPE_BF16, N, D, ptr<float>(out), st);
  });
  return out;
}

Tensor rademacher(int64_t rows, int64_t cols, uint64_t seed, uint64_t offset, const Tensor& like) {
  c10::cuda::CUDAGuard guard(like.device());
  Tensor out = empty({rows, cols}, at::kFloat, like);
  invoke("exact_rademacher", {rows * cols * 4},
         [&](void* st) { return lib.exact_rademacher(seed, offset, rows, cols, ptr<float>(out), st); });
  return out;
}

// fp32 rows of any length, k up to 512 as long as the pipeline stages of a [128 x 32] A tile and a [k x 32] sign tile fit
bool rp_supported(int64_t D, int64_t k) {
  const int64_t kpad = (k + 15) / 16 * 16, stage = 128 * 128 + kpad * 128;
  return kpad <= 512 && 200 * 1024 / stage >= (D % 4 ? 3 : 2);
}

Packed rp_quantize_pack(const Tensor& x, const Tensor& R, int64_t bits, uint64_t seed, uint64_t offset, int64_t row_offset,
                        Tensor* projection) {
  if (!x.is_cuda() || x.dim() != 2 || x.stride(1) != 1 || x.stride(0) < x.size(1)) check_tensor(x, "data", 2);   // any pitch
  check_type(x.scalar_type() == at::kFloat, "data");
  check_tensor(R, "R", 2);
  check_type(R.scalar_type() == at::kFloat, "R");
  check_bits(bits);
  same_device(x, R);
  const int64_t N = x.size(0), D = x.size(1), k = R.size(1);
  if (R.size(0) != D) throw std::runtime_error("R must be [D, k]");
  if (!rp_supported(D, k)) throw LibraryError("rp_quantize_pack: unsupported shape (needs fp32 and k <= 512)");
  c10::cuda::CUDAGuard guard(x.device());
  if (projection) *projection = empty({N, k}, at::kFloat, x);
  Tensor ws = empty({lib.exact_rp_workspace_bytes(D, k)}, at::kByte, x);
  const int64_t bytes = lib.exact_packed_bytes(N, k, (int)bits);
  Packed q{empty({bytes + 1}, at::kChar, x), empty({N}, at::kBFloat16, x), empty({N}, at::kBFloat16, x)};
  invoke("exact_rp_quantize_pack", {N * D * 4 + D * k * 4 + bytes + 4 * N}, [&](void* st) {
    return lib.exact_rp_quantize_pack_rows(ptr<float>(x), N, D, N > 1 ? x.stride(0) : D, ptr<float>(R), k, (int)bits, seed, offset, row_offset, ptr(ws),
                                      ptr<uint8_t>(q.codes), ptr<uint16_t>(q.scale), ptr<uint16_t>(q.mn),
                                      projection ? ptr<float>(*projection) : nullptr, st);
  });
  mark_status(x);
  return q;
}

bool linear_supported(const Tensor& a) {
  return a.is_cuda() && a.scalar_type() == at::kFloat && a.dim() == 2 && a.size(0) >= 1024;
}

// Rows that start on 16-byte boundaries, as tensor maps want them: `a`, or a copy with its rows zero-padded to whole
// 16-byte pieces (one pass; a layer that multiplies the same rows twice makes the copy once and passes it on).
Tensor rows16(const Tensor& a) {
  if (a.stride(1) == 1 && a.stride(0) % 4 == 0 && a.stride(0) >= a.size(1) && reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0)
    return a;
  const Tensor rows = a.stride(1) == 1 && a.stride(0) >= a.size(1) ? a : a.contiguous();
  return std::get<0>(rows_scale_colsum(rows, {}, true, false)).narrow(1, 0, a.size(1));
}

Tensor linear(const Tensor& a_, const Tensor& w_, const OptTensor& bias_, const OptTensor& a2_, const OptTensor& w2_,
              const OptTensor& out_, bool accumulate, int64_t k_chunk, const OptTensor& addend_) {
  c10::cuda::CUDAGuard guard(a_.device());
  const int64_t M = a_.size(0), K = a_.size(1), N = w_.size(0);
  const Tensor a = rows16(a_), w = w_;
  Tensor a2, w2, bias;
  int64_t K2 = 0;
  if (a2_) {
    K2 = a2_->size(1);
    a2 = rows16(*a2_);
    w2 = *w2_;
  }
  if (bias_) bias = bias_->contiguous();
  Tensor out = out_ ? *out_ : empty({M, N}, at::kFloat, a);
  const OptTensor addend = addend_ ? addend_ : out_ && accumulate ? OptTensor(out) : OptTensor();
  if (out.size(0) != M || out.size(1) != N || out.stride(1) != 1) throw std::runtime_error("linear: out does not fit");
  for (int64_t n0 = 0; n0 < N; n0 += 256) {
    const int64_t n = std::min<int64_t>(N - n0, 256);
    Tensor ws = empty({lib.exact_linear_workspace_bytes(n, K, K2)}, at::kByte, a);
    const float* wb = ptr<float>(w) + n0 * w.stride(0);
    const float* w2b = K2 ? ptr<float>(w2) + n0 * w2.stride(0) : nullptr;
    float* cb = ptr<float>(out) + n0;
    CallInfo info;
    info.bytes = 4 * (M * (K + K2) + n * (K + K2) + M * n * (addend ? 2 : 1));
    info.flops = 6.0 * (double)M * (double)(K + K2) * (double)n;
    // two kernels with different rates: timed under two names
    invoke(k_chunk > 0 ? "exact_linear_forward" : "exact_linear_forward_tf32", info, [&](void* st) {
      return lib.exact_linear_forward_strided(ptr<float>(a), M, K, a.stride(0), wb, w.stride(0), w.stride(1), K2 ? ptr<float>(a2) : nullptr, K2,
                                      K2 ? a2.stride(0) : 0, w2b, K2 ? w2.stride(0) : 0, K2 ? w2.stride(1) : 1, n,
                                      bias.defined() ? ptr<float>(bias) + n0 : nullptr,
                                              addend ? ptr<float>(addend) + n0 : nullptr, addend ? addend->stride(0) : 0,
                                              k_chunk, nullptr, ptr(ws),
                                              cb, out.stride(0), st);
    });
  }
  mark_status(a);
  return out;
}

// The one rule of which weight gradients the kernel forms; the others are unpacked and go to rows_reduce_mm.
bool grad_weight_takes(const Tensor& g) {
  return g.is_cuda() && g.scalar_type() == at::kFloat && g.dim() == 2 && g.size(0) > 0 && g.size(1) <= 256;
}

// g^T x with the reduction over rows cut into products that one batched library GEMM computes in parallel: a single one leaves
// most SMs idle on this shape, and its sums are longer.
Tensor rows_reduce_mm(const Tensor& g, const Tensor& x, int64_t batches) {
  const int64_t M = g.size(0);
  if (!g.is_cuda() || M < 64 * batches || !g.is_contiguous() || !x.is_contiguous()) return at::mm(g.t(), x);
  const int64_t rows = M / batches * batches;
  Tensor out = at::bmm(g.narrow(0, 0, rows).view({batches, -1, g.size(1)}).transpose(1, 2), x.narrow(0, 0, rows).view({batches, -1, x.size(1)})).sum(0);
  if (rows < M) out.addmm_(g.narrow(0, rows, M - rows).t(), x.narrow(0, rows, M - rows));
  return out;
}

// g^T . dequantise(q0 | q1): [O, pad16(k0) + pad16(k1)] with the second block from column pad16(k0) on.
Tensor grad_weight(const Tensor& g_, int64_t bits, const Packed& q0, int64_t k0, const Packed* q1, int64_t k1) {
  c10::cuda::CUDAGuard guard(g_.device());
  Tensor g = g_.size(1) % 4 ? at::constant_pad_nd(g_, {0, 4 - g_.size(1) % 4}) : g_.contiguous();
  if (reinterpret_cast<uintptr_t>(g.data_ptr()) % 16) g = g.clone();      // a view off the 16 bytes that a tensor map wants
  const int64_t N = g.size(0), O = g.size(1);
  const int64_t kpad = (k0 + 15) / 16 * 16 + (q1 ? (k1 + 15) / 16 * 16 : 0);
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  const int64_t ws_bytes = lib.exact_grad_weight_workspace_bytes(O, kpad, sms);
  Tensor ws = empty({ws_bytes}, at::kByte, g), out = empty({O, kpad}, at::kFloat, g);
  CallInfo info;
  info.bytes = 4 * N * O + (N * (k0 + (q1 ? k1 : 0)) * bits) / 8 + 4 * N * (q1 ? 2 : 1);
  info.flops = 2.0 * (double)N * (double)O * (double)kpad;
  invoke("exact_grad_weight_from_packed", info, [&](void* st) {
    return lib.exact_grad_weight_from_packed(
        ptr<float>(g), N, O, ptr<uint8_t>(q0.codes), ptr<uint16_t>(q0.scale), ptr<uint16_t>(q0.mn), k0,
        q1 ? ptr<uint8_t>(q1->codes) : nullptr, q1 ? ptr<uint16_t>(q1->scale) : nullptr, q1 ? ptr<uint16_t>(q1->mn) : nullptr,
        q1 ? k1 : 0, (int)bits, ptr(ws), ws_bytes, ptr<float>(out), kpad, st);
  });
  mark_status(g);
  return g_.size(1) != O ? out.narrow(0, 0, g_.size(1)) : out;
}

std::tuple<Tensor, Tensor> rows_scale_colsum(const Tensor& g, const OptTensor& rowscale, bool want_scaled, bool want_colsum) {
  c10::cuda::CUDAGuard guard(g.device());
  const int64_t N = g.size(0), K = g.size(1), Kout = want_scaled ? (K + 3) / 4 * 4 : K;
  Tensor out, colsum, ws;
  int64_t ws_bytes = 0;
  if (want_scaled) out = empty({N, Kout}, at::kFloat, g);
  if (want_colsum) {
    colsum = empty({K}, at::kFloat, g);
    ws_bytes = lib.exact_rows_scale_colsum_workspace_bytes(Kout);
    ws = empty({ws_bytes}, at::kByte, g);
  }
  invoke("exact_rows_scale_colsum", {4 * N * K + (want_scaled ? 4 * N * Kout : 0)}, [&](void* st) {
    return lib.exact_rows_scale_colsum(ptr<float>(g), N, K, g.stride(0), ptr<float>(rowscale),
                                       want_scaled ? ptr<float>(out) : nullptr, Kout, Kout,
                                       want_colsum ? ptr<float>(colsum) : nullptr, want_colsum ? ptr(ws) : nullptr, ws_bytes, st);
  });
  return {out, colsum};
}

std::tuple<Tensor, Tensor, Tensor> rows_scale_copy_colsum(const Tensor& g, const OptTensor& rowscale, bool want_colsum) {
  c10::cuda::CUDAGuard guard(g.device());
  const int64_t N = g.size(0), K = g.size(1), Kout = (K + 3) / 4 * 4;
  Tensor out = empty({N, Kout}, at::kFloat, g), copy = empty({N, Kout}, at::kFloat, g), colsum, ws;
  int64_t ws_bytes = 0;
  if (want_colsum) {
    colsum = empty({K}, at::kFloat, g);
    ws_bytes = lib.exact_rows_scale_colsum_workspace_bytes(Kout);
    ws = empty({ws_bytes}, at::kByte, g);
  }
  invoke("exact_rows_scale_colsum", {4 * N * K + 8 * N * Kout}, [&](void* st) {
    return lib.exact_rows_scale_copy_colsum(ptr<float>(g), N, K, g.stride(0), ptr<float>(rowscale), ptr<float>(out), ptr<float>(copy),
                                            Kout, Kout, want_colsum ? ptr<float>(colsum) : nullptr, want_colsum ? ptr(ws) : nullptr,
                                            ws_bytes, st);
  });
  return {out, copy, colsum};
}

std::tuple<Tensor, Tensor> rows_half_colsum(const Tensor& g, bool want_colsum) {
  c10::cuda::CUDAGuard guard(g.device());
  const int64_t N = g.size(0), K = g.size(1), Kout = (K + 7) / 8 * 8;
  Tensor out = empty({N, Kout}, at::kHalf, g), colsum, ws;
  int64_t ws_bytes = 0;
  if (want_colsum) {
    colsum = empty({K}, at::kFloat, g);
    ws_bytes = lib.exact_rows_scale_colsum_workspace_bytes(Kout);
    ws = empty({ws_bytes}, at::kByte, g);
  }
  invoke("exact_rows_half_colsum", {4 * N * K + 2 * N * Kout}, [&](void* st) {
    return lib.exact_rows_half_colsum(ptr<float>(g), N, K, g.stride(0), ptr(out), Kout, Kout, want_colsum ? ptr<float>(colsum) : nullptr,
                                      want_colsum ? ptr(ws) : nullptr, ws_bytes, st);
  });
  return {out, colsum};
}

std::tuple<Tensor, Tensor, Tensor> bn_forward(const Tensor& x, const OptTensor& weight_, const OptTensor& bias_,
                                              const OptTensor& running_mean, const OptTensor& running_var, double momentum,
                                              double eps) {
  c10::cuda::CUDAGuard guard(x.device());
  OptTensor weight, bias;
  if (weight_) weight = weight_->detach().contiguous();
  if (bias_) bias = bias_->detach().contiguous();
  const int64_t N = x.size(0), D = x.size(1), ws_bytes = lib.exact_bn_forward_workspace_bytes(D);
  Tensor ws = empty({ws_bytes}, at::kByte, x), y = empty({N, D}, at::kFloat, x), mean = empty({D}, at::kFloat, x),
         invstd = empty({D}, at::kFloat, x);
  invoke("exact_bn_forward", {12 * N * D}, [&](void* st) {
    return lib.exact_bn_forward(ptr<float>(x), N, D, ptr<float>(weight), ptr<float>(bias), ptr<float>(running_mean),
                                ptr<float>(running_var), (float)momentum, (float)eps, ptr(ws), ws_bytes, ptr<float>(y),
                                ptr<float>(mean), ptr<float>(invstd), st);
  });
  return {y, mean, invstd};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> bn_act_forward(const Tensor& x, const OptTensor& weight_, const OptTensor& bias_,
                                                          const OptTensor& running_mean, const OptTensor& running_var,
                                                          double momentum, double eps, double p, uint64_t seed, uint64_t offset,
                                                          int64_t index_offset) {
  c10::cuda::CUDAGuard guard(x.device());
  OptTensor weight, bias;
  if (weight_) weight = weight_->detach().contiguous();
  if (bias_) bias = bias_->detach().contiguous();
  const int64_t N = x.size(0), D = x.size(1), ws_bytes = lib.exact_bn_forward_workspace_bytes(D);
  Tensor ws = empty({ws_bytes}, at::kByte, x), out = empty({N, D}, at::kFloat, x), mean = empty({D}, at::kFloat, x),
         invstd = empty({D}, at::kFloat, x), mask = empty({lib.exact_mask_words(N * D)}, at::kInt, x);
  invoke("exact_bn_act_forward", {12 * N * D + N * D / 8}, [&](void* st) {
    return lib.exact_bn_act_forward(ptr<float>(x), N, D, ptr<float>(weight), ptr<float>(bias), ptr<float>(running_mean),
                                    ptr<float>(running_var), (float)momentum, (float)eps, (float)p, seed, offset, index_offset,
                                    ptr(ws), ws_bytes, ptr<float>(out), ptr<uint32_t>(mask), ptr<float>(mean), ptr<float>(invstd),
                                    st);
  });
  return {out, mask, mean, invstd};
}

std::tuple<Tensor, Tensor, Tensor> bn_backward(const Tensor& g_, const Packed& q, int64_t bits, const OptTensor& weight_,
                                               const Tensor& mean_, const Tensor& invstd_, bool train, bool want_input,
                                               bool want_weight, bool want_bias, const OptTensor& mask, double p) {
  c10::cuda::CUDAGuard guard(g_.device());
  const Tensor g = g_.contiguous(), mean = mean_.to(at::kFloat).contiguous(), invstd = invstd_.to(at::kFloat).contiguous();
  OptTensor weight;
  if (weight_) weight = weight_->detach().to(at::kFloat).contiguous();
  const int64_t N = g.size(0), D = g.size(1), ws_bytes = lib.exact_bn_backward_workspace_bytes(D);
  Tensor ws = empty({ws_bytes}, at::kByte, g), gi, gw, gb;
  if (want_input) gi = empty({N, D}, at::kFloat, g);
  if (want_weight) gw = empty({D}, at::kFloat, g);
  if (want_bias) gb = empty({D}, at::kFloat, g);
  const int64_t pass = N * D * 4 + lib.exact_packed_bytes(N, D, (int)bits) + 4 * N;
  const bool both = want_input && (train || want_weight || want_bias);
  if (mask) {
    invoke("exact_bn_act_backward_from_packed", {(both ? 2 : 1) * (pass + N * D / 8) + (want_input ? N * D * 4 : 0)}, [&](void* st) {
      return lib.exact_bn_act_backward_from_packed(ptr<float>(g), ptr<uint32_t>(*mask), (float)p, N, D, ptr<uint8_t>(q.codes),
                                                   (int)bits, ptr<uint16_t>(q.scale), ptr<uint16_t>(q.mn), ptr<float>(weight),
                                                   ptr<float>(mean), ptr<float>(invstd), ptr(ws), ws_bytes,
                                                   want_input ? ptr<float>(gi) : nullptr, want_weight ? ptr<float>(gw) : nullptr,
                                                   want_bias ? ptr<float>(gb) : nullptr, st);
    });
    return {gi, gw, gb};
  }
  invoke("exact_bn_backward_from_packed", {(both ? 2 : 1) * pass + (want_input ? N * D * 4 : 0)}, [&](void* st) {
    return lib.exact_bn_backward_from_packed(ptr<float>(g), N, D, ptr<uint8_t>(q.codes), (int)bits, ptr<uint16_t>(q.scale),
                                             ptr<uint16_t>(q.mn), ptr<float>(weight), ptr<float>(mean), ptr<float>(invstd),
                                             train ? 1 : 0, ptr(ws), ws_bytes, want_input ? ptr<float>(gi) : nullptr,
                                             want_weight ? ptr<float>(gw) : nullptr, want_bias ? ptr<float>(gb) : nullptr, st);
  });
  return {gi, gw, gb};
}

std::tuple<Tensor, Tensor> act_forward(int64_t op, const Tensor& x, double param, const OptTensor& uniforms, uint64_t seed,
                                       uint64_t offset, int64_t index_offset) {
  check_tensor(x, "input", -1);
  check_type(x.scalar_type() == at::kFloat || x.scalar_type() == at::kHalf, "input");
  if (uniforms) {
    check_tensor(*uniforms, "uniforms", -1);
    check_type(uniforms->scalar_type() == at::kFloat, "uniforms");
    if (uniforms->numel() != x.numel()) throw std::runtime_error("uniforms must have the shape of input");
    same_device(x, *uniforms);
    seed = offset = 0;
  }
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t n = x.numel();
  Tensor out = empty(x.sizes(), x.scalar_type(), x), mask = empty({lib.exact_mask_words(n)}, at::kInt, x);
  uint32_t* m = ptr<uint32_t>(mask);
  const float p = (float)param;
  if (x.scalar_type() == at::kHalf) {
    invoke("exact_act_quantized_forward_f16", {4 * n + n / 8}, [&](void* st) {
      return lib.exact_act_quantized_forward_f16((int)op, ptr<uint16_t>(x), n, p, ptr<float>(uniforms), seed, offset, index_offset,
                                                 ptr<uint16_t>(out), m, st);
    });
    return {out, mask};
  }
  const CallInfo info{8 * n + n / 8};
  const float* xi = ptr<float>(x);
  float* o = ptr<float>(out);
  switch (op) {
    case ACT_RELU:
      invoke("exact_act_quantized_relu_forward", info, [&](void* st) { return lib.exact_act_quantized_relu_forward(xi, n, o, m, st); });
      break;
    case ACT_LEAKY_RELU:
      invoke("exact_act_quantized_leaky_relu_forward", info,
             [&](void* st) { return lib.exact_act_quantized_leaky_relu_forward(xi, n, p, o, m, st); });
      break;
    case ACT_DROPOUT:
      invoke("exact_act_quantized_dropout_forward", info, [&](void* st) {
        return lib.exact_act_quantized_dropout_forward(xi, n, p, ptr<float>(uniforms), seed, offset, index_offset, o, m, st);
      });
      break;
    default:
      invoke("exact_act_quantized_relu_dropout_forward", info, [&](void* st) {
        return lib.exact_act_quantized_relu_dropout_forward(xi, n, p, ptr<float>(uniforms), seed, offset, index_offset, o, m, st);
      });
  }
  return {out, mask};
}

Tensor act_backward(int64_t op, const Tensor& g_, const Tensor& mask, double param) {
  c10::cuda::CUDAGuard guard(g_.device());
  const Tensor g = g_.contiguous();
  const int64_t n = g.numel();
  Tensor out = empty(g.sizes(), g.scalar_type(), g);
  const uint32_t* m = ptr<uint32_t>(mask);
  const float p = (float)param;
  if (g.scalar_type() == at::kHalf) {
    if (op == ACT_RELU_DROPOUT) op = ACT_DROPOUT;   // one mask: the dropout's backward with it
    invoke("exact_act_quantized_backward_f16", {4 * n + n / 8}, [&](void* st) {
      return lib.exact_act_quantized_backward_f16((int)op, ptr<uint16_t>(g), m, n, p, ptr<uint16_t>(out), st);
    });
    return out;
  }
  const CallInfo info{8 * n + n / 8};
  const float* gi = ptr<float>(g);
  float* o = ptr<float>(out);
  if (op == ACT_RELU)
    invoke("exact_act_quantized_relu_backward", info, [&](void* st) { return lib.exact_act_quantized_relu_backward(gi, m, n, o, st); });
  else if (op == ACT_LEAKY_RELU)
    invoke("exact_act_quantized_leaky_relu_backward", info,
           [&](void* st) { return lib.exact_act_quantized_leaky_relu_backward(gi, m, n, p, o, st); });
  else
    invoke("exact_act_quantized_dropout_backward", info,
           [&](void* st) { return lib.exact_act_quantized_dropout_backward(gi, m, n, p, o, st); });
  return out;
}

const RowPlan::Pieces& RowPlan::pieces(const Tensor& rowptr, const Tensor& col) const {
  std::lock_guard<std::mutex> lock(mu);
  if (cut) return *cut;
  Pieces p;
  const int64_t M = rowptr.size(0) - 1, t = threshold;
  if (t > 0 && M > 0) {
    const Tensor begin = rowptr.narrow(0, 0, M), end = rowptr.narrow(0, 1, M);
    const Tensor rows = at::nonzero((end - begin).gt(t)).flatten();
    p.n_long = rows.size(0);
    if (p.n_long) {
      const Tensor b = begin.index_select(0, rows).to(at::kLong), e = end.index_select(0, rows).to(at::kLong);
      const Tensor count = at::floor_divide(e - b + (t - 1), t), ptr = at::cumsum(count, 0);
      p.n = ptr[-1].item<int64_t>();
      const Tensor which = at::repeat_interleave(count, std::optional<int64_t>(p.n)), first = ptr - count;   // piece -> long row
      const Tensor within = at::arange(p.n, count.options()) - first.index_select(0, which);
      const Tensor pb = b.index_select(0, which) + within * t, pe = at::minimum(pb + t, e.index_select(0, which));
      const Tensor by_col = at::argsort(col.index_select(0, pb), /*stable=*/true);
      p.row = rows.index_select(0, which.index_select(0, by_col)).to(at::kInt);
      p.begin = pb.index_select(0, by_col);
      p.end = pe.index_select(0, by_col);
      p.slot = by_col.to(at::kInt);
      p.long_row = rows.to(at::kInt);
      p.long_ptr = at::constant_pad_nd(ptr, {1, 0}).to(at::kInt);
    }
  }
  cut = p;
  return *cut;
}
const Tensor& RowPlan::row_order(const Tensor& rowptr) const {
  std::lock_guard<std::mutex> lock(mu);
  if (!order.defined()) {
    const int64_t M = rowptr.size(0) - 1;
    const Tensor deg = rowptr.narrow(0, 1, M) - rowptr.narrow(0, 0, M);
    order = at::argsort(deg, /*stable=*/true, /*dim=*/-1, /*descending=*/true).to(at::kInt);
  }
  return order;
}
int64_t RowPlan::n_long_f16(const Tensor& rowptr) const {
  std::lock_guard<std::mutex> lock(mu);
  if (n_f16 < 0) {
    const int64_t M = rowptr.size(0) - 1;
    n_f16 = threshold_f16 > 0
                ? (rowptr.narrow(0, 1, M) - rowptr.narrow(0, 0, M)).gt(threshold_f16).sum().item<int64_t>() : 0;
  }
  return n_f16;
}

Tensor spmm(const Tensor& rowptr, const Tensor& colt, const RowPlan& a, const OptTensor& value_, const Tensor& mat_, bool mean,
            const OptTensor& bias_) {
  const Tensor mat = mat_.contiguous();
  same_device(rowptr, mat);
  same_device(colt, mat);
  c10::cuda::CUDAGuard guard(mat.device());
  const int64_t M = rowptr.size(0) - 1, K = mat.size(1), nnz = colt.size(0);
  const int ib = colt.scalar_type() == at::kInt ? 4 : 8;
  const int red = mean ? EXACT_REDUCE_MEAN : EXACT_REDUCE_SUM;
  const void *rp = ptr(rowptr), *col = ptr(colt);
  OptTensor bias;
  if (bias_) bias = bias_->detach().to(at::kFloat).contiguous();
  if (mat.scalar_type() == at::kHalf) {
    // the reference's half instantiation (spmm_cuda.cu:142): every step rounded to half, rows in CSR order
    OptTensor value;
    if (value_) value = value_->detach().to(at::kHalf).contiguous();
    Tensor out = empty({M, K}, bias ? at::kFloat : at::kHalf, mat), src = mat;
    const int64_t ldm = (K + 7) / 8 * 8;
    if (ldm != K) {   // rows in whole 16-byte pieces: the copy is read and written once, the gathers nnz / N times
      src = empty({mat.size(0), ldm}, at::kHalf, mat);
      src.narrow(1, 0, K).copy_(mat);
    }
    const int32_t* order = ptr<int32_t>(a.row_order(rowptr));
    const int64_t n_long = a.n_long_f16(rowptr);
    invoke("exact_spmm_f16", {nnz * (2 * K + ib) + 2 * M * K}, [&](void* st) {
      return lib.exact_spmm_f16_planned(rp, col, ib, ptr(value), ptr(src), ldm, M, K, red, order, a.threshold_f16,
                                        n_long ? order : nullptr, n_long, ptr<float>(bias), ptr(out), st);
    });
    return out;
  }
  OptTensor value;
  if (value_) value = value_->detach().to(at::kFloat).contiguous();
  Tensor out = empty({M, K}, at::kFloat, mat);
  const int64_t index_bytes = nnz * (ib + (value ? 4 : 0)) + (M + 1) * ib;
  CallInfo info;
  info.bytes = mat.size(0) * K * 4 + index_bytes + M * K * 4;   // what must cross HBM at least once
  info.l2_bytes = nnz * K * 4 + index_bytes + M * K * 4;        // what the gathers request when no source row is reused
  info.edge_columns = nnz * K;
  // Rows of whole 16-byte pieces: an odd width is gathered element by element in 32-column passes over the graph, an even one in
  // pairs.  The padded copy is one pass over the operand, which a call of a few microseconds does not repay; a wide odd
  // operand of a small graph is bound by latency, and its many narrow passes hide that better (18.7 M edges x 47 columns
  // 598 -> 390 us, x 90 922 -> 649, x 145 1,452 -> 1,229; 0.46 M x 47 56 -> 39, x 90 81 -> 70, x 145 88 -> 103).
  int64_t ldm = K;
  Tensor src = mat;
  if (K % 4 && nnz >= 2 * mat.size(0) && nnz * K >= (K <= 64 || K % 2 == 0 ? 1LL << 22 : 1LL << 27)) {
    ldm = (K + 3) / 4 * 4;
    src = std::get<0>(rows_scale_colsum(mat, {}, true, false));
  }
  const RowPlan::Pieces& pc = a.pieces(rowptr, colt);
  Tensor scratch;
  if (pc.n) scratch = empty({pc.n, ldm}, at::kFloat, mat);
  float* sc = pc.n ? ptr<float>(scratch) : nullptr;
  const int32_t *prow = nullptr, *pslot = nullptr, *lrow = nullptr, *lptr = nullptr;
  const int64_t *pb = nullptr, *pe = nullptr;
  if (pc.n) {
    prow = ptr<int32_t>(pc.row); pslot = ptr<int32_t>(pc.slot); lrow = ptr<int32_t>(pc.long_row); lptr = ptr<int32_t>(pc.long_ptr);
    pb = ptr<int64_t>(pc.begin); pe = ptr<int64_t>(pc.end);
  }
  const bool narrow = ldm <= 64 && ldm % 4 == 0 && M > 0;
  const int32_t* order = M > 0 ? ptr<int32_t>(a.row_order(rowptr)) : nullptr;
  invoke(narrow ? "exact_spmm_split_routed" : pc.n ? "exact_spmm_split" : "exact_spmm", info, [&](void* st) {
    return lib.exact_spmm_planned(rp, col, ib, ptr<float>(value), ptr<float>(src), ldm, M, K, red, pc.n ? a.threshold : 0, prow, pb, pe,
                                  pslot, pc.n, lrow, lptr, pc.n_long, sc, order, ptr<float>(bias), ptr<float>(out), st);
  });
  return out;
}

std::tuple<Tensor, Tensor> spmm_minmax(const Tensor& rowptr, const Tensor& col, const RowPlan& plan, const OptTensor& value_,
                                       const Tensor& mat_, bool is_max) {
  const Tensor mat = mat_.contiguous();
  check_type(mat.scalar_type() == at::kFloat, "mat");
  same_device(rowptr, mat);
  same_device(col, mat);
  c10::cuda::CUDAGuard guard(mat.device());
  OptTensor value;
  if (value_) value = value_->detach().to(at::kFloat).contiguous();
  const int64_t M = rowptr.size(0) - 1, K = mat.size(1), nnz = col.size(0);
  const int ib = col.scalar_type() == at::kInt ? 4 : 8;
  Tensor out = empty({M, K}, at::kFloat, mat), arg = empty({M, K}, col.scalar_type(), mat), scratch;
  const RowPlan::Pieces& pc = plan.pieces(rowptr, col);
  if (pc.n) scratch = empty({lib.exact_spmm_minmax_scratch_bytes(pc.n, K)}, at::kByte, mat);
  invoke("exact_spmm_minmax", {nnz * (K * 4 + ib) + M * K * (4 + ib)}, [&](void* st) {
    return lib.exact_spmm_minmax_planned(ptr(rowptr), ptr(col), ib, ptr<float>(value), ptr<float>(mat), M, K, nnz, is_max ? 1 : 0,
                                         pc.n ? plan.threshold : 0, pc.n ? ptr<int64_t>(pc.begin) : nullptr,
                                         pc.n ? ptr<int64_t>(pc.end) : nullptr, pc.n ? ptr<int32_t>(pc.slot) : nullptr, pc.n,
                                         pc.n ? ptr<int32_t>(pc.long_row) : nullptr, pc.n ? ptr<int32_t>(pc.long_ptr) : nullptr,
                                         pc.n_long, pc.n ? ptr(scratch) : nullptr, ptr<float>(out), ptr(arg), st);
  });
  return {out, arg};
}

std::tuple<Tensor, Tensor> spmm_minmax_backward(const Tensor& col, const OptTensor& value_, const OptTensor& mat, const Tensor& arg,
                                                const Tensor& grad_, bool need_value, bool need_mat, int64_t mat_rows) {
  const Tensor grad = grad_.contiguous();
  c10::cuda::CUDAGuard guard(grad.device());
  OptTensor value;
  if (value_) value = value_->detach().to(at::kFloat).contiguous();
  const int64_t M = grad.size(0), K = grad.size(1), nnz = col.size(0);
  const int ib = col.scalar_type() == at::kInt ? 4 : 8;
  Tensor gv, gm;
  const auto opts = grad.options().requires_grad(false);
  if (need_value) gv = at::zeros({nnz}, opts);
  if (need_mat) gm = at::zeros({mat_rows, K}, opts);
  invoke("exact_spmm_minmax_backward", {M * K * (8 + ib) + (need_mat ? mat_rows * K * 4 : 0)}, [&](void* st) {
    return lib.exact_spmm_minmax_backward(ptr(col), ib, ptr<float>(value), ptr<float>(mat), ptr(arg), ptr<float>(grad), M, K, nnz,
                                          need_mat ? ptr<float>(gm) : nullptr, need_value ? ptr<float>(gv) : nullptr, st);
  });
  return {gv, gm};
}

std::tuple<Tensor, Tensor> spmm_weighted_backward(const Csr& t, const Tensor& perm, const OptTensor& fw_rowptr, const Tensor& mat_,
                                                  const Tensor& grad_) {
  const Tensor mat = mat_.contiguous(), grad = grad_.contiguous();
  check_type(mat.scalar_type() == at::kFloat && grad.scalar_type() == at::kFloat, "mat or grad");
  check_type(perm.scalar_type() == t.col.scalar_type() && (!fw_rowptr || fw_rowptr->scalar_type() == t.col.scalar_type()), "perm or rowptr");
  same_device(t.rowptr, mat);
  same_device(t.col, grad);
  same_device(perm, grad);
  c10::cuda::CUDAGuard guard(mat.device());
  const int64_t M = t.rowptr.size(0) - 1, K = mat.size(1), nnz = t.col.size(0);
  const int ib = t.col.scalar_type() == at::kInt ? 4 : 8;
  const RowPlan::Pieces& pc = t.plan->pieces(t.rowptr, t.col);
  Tensor gm = empty({M, K}, at::kFloat, mat), gv = empty({nnz}, at::kFloat, mat), scratch;
  if (pc.n) scratch = empty({pc.n, K}, at::kFloat, mat);
  CallInfo info;
  info.bytes = 4 * K * (2 * M + grad.size(0)) + nnz * (2 * ib + 8) + (M + 1) * ib;
  info.l2_bytes = nnz * K * 4 + info.bytes;
  info.edge_columns = nnz * K;
  const int32_t* order = M > 0 ? ptr<int32_t>(t.plan->row_order(t.rowptr)) : nullptr;
  invoke("exact_spmm_weighted_backward", info, [&](void* st) {
    return lib.exact_spmm_weighted_backward(
        ptr(t.rowptr), ptr(t.col), ptr<float>(*t.value), ptr(perm), ptr(fw_rowptr), ib, ptr<float>(mat), ptr<float>(grad), M, K,
        pc.n ? t.plan->threshold : 0, pc.n ? ptr<int32_t>(pc.row) : nullptr, pc.n ? ptr<int64_t>(pc.begin) : nullptr,
        pc.n ? ptr<int64_t>(pc.end) : nullptr, pc.n ? ptr<int32_t>(pc.slot) : nullptr, pc.n, pc.n ? ptr<int32_t>(pc.long_row) : nullptr,
        pc.n ? ptr<int32_t>(pc.long_ptr) : nullptr, pc.n_long, pc.n ? ptr<float>(scratch) : nullptr, order, ptr<float>(gm), ptr<float>(gv),
        st);
  });
  return {gm, gv};
}

Tensor spmm_value_backward(const Tensor& row, const Tensor& rowptr, const Tensor& col, const Tensor& mat_, const Tensor& grad_,
                           bool mean) {
  const Tensor mat = mat_.contiguous(), grad = grad_.contiguous();
  check_type(mat.scalar_type() == at::kFloat && grad.scalar_type() == at::kFloat, "mat or grad");
  check_type(row.scalar_type() == col.scalar_type() && rowptr.scalar_type() == col.scalar_type(), "row, rowptr or col");
  same_device(row, mat);
  same_device(col, grad);
  c10::cuda::CUDAGuard guard(mat.device());
  const int64_t E = col.size(0), K = mat.size(1);
  const int ib = col.scalar_type() == at::kInt ? 4 : 8;
  Tensor out = empty({E}, at::kFloat, mat);
  invoke("exact_spmm_value_bw", {E * (8 * K + 2 * ib + 4)}, [&](void* st) {
    return lib.exact_spmm_value_bw(ptr(row), ptr(rowptr), ptr(col), ib, ptr<float>(mat), ptr<float>(grad), E, K,
                                   mean ? EXACT_REDUCE_MEAN : EXACT_REDUCE_SUM, ptr<float>(out), st);
  });
  return out;
}

}  // namespace exb

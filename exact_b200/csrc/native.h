// Host path of the hot ops: argument checks, allocation and launch in C++ on torch tensors.
//
// The Python layer calls these instead of binding the C ABI entry by entry with ctypes: a call cost 16 - 20 us there
// (tensor attributes, device and stream look-ups, four allocations, the ctypes conversion of up to 25 arguments), 2 - 4 us
// here, and a training step of a small graph is nothing but such calls.  The C ABI stays the boundary: every kernel is
// launched through the functions of exact_b200.h, looked up in the library that _lib.py names.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <memory>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "exact_b200.h"

namespace exb {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

struct LibraryError : std::runtime_error {   // becomes exact_b200.ExactB200Error
  using std::runtime_error::runtime_error;
};

// ---- the C ABI, resolved at run time ----------------------------------------------------------------
#define EXB_FUNCTIONS(X)                                                                                              \
  X(exact_last_error) X(exact_packed_bytes) X(exact_quantize_pack) X(exact_quantize_pack_f16)                         \
  X(exact_unpack_single_precision) X(exact_unpack_single_precision_f16) X(exact_mask_words)                           \
  X(exact_act_quantized_relu_forward) X(exact_act_quantized_relu_backward) X(exact_act_quantized_leaky_relu_forward)  \
  X(exact_act_quantized_leaky_relu_backward) X(exact_act_quantized_dropout_forward)                                   \
  X(exact_act_quantized_dropout_backward) X(exact_act_quantized_relu_dropout_forward)                                 \
  X(exact_act_quantized_forward_f16) X(exact_act_quantized_backward_f16) X(exact_spmm_planned)                        \
  X(exact_spmm_f16_planned) X(exact_rows_scale_colsum_workspace_bytes)                     \
  X(exact_rows_scale_colsum) X(exact_bn_forward_workspace_bytes) X(exact_bn_forward) X(exact_rows_half_colsum) \
  X(exact_rows_scale_copy_colsum) X(exact_quantize_pack_rows) X(exact_rp_quantize_pack_rows)                          \
  X(exact_bn_backward_workspace_bytes) X(exact_bn_backward_from_packed) X(exact_bn_act_forward)                       \
  X(exact_bn_act_backward_from_packed)                                                                                \
  X(exact_rp_workspace_bytes) X(exact_rademacher) X(exact_grad_weight_workspace_bytes)      \
  X(exact_grad_weight_from_packed) X(exact_linear_workspace_bytes) X(exact_linear_forward_strided)                            \
  X(exact_spmm_minmax_scratch_bytes) X(exact_spmm_minmax_planned) X(exact_spmm_minmax_backward)                       \
  X(exact_spmm_value_bw) X(exact_spmm_weighted_backward) X(exact_status_peek)

struct Library {
#define EXB_POINTER(name) decltype(&::name) name = nullptr;
  EXB_FUNCTIONS(EXB_POINTER)
#undef EXB_POINTER
};
extern Library lib;

// ---- launch accounting (mirrored by _lib.LAUNCHES, _lib.TIMER and _lib.HOST_CLOCK) ---------------------
struct TimedCall {
  const char* name;
  cudaEvent_t begin, end;
  int64_t bytes;
  int64_t l2_bytes, edge_columns;   // -1: not given
  double flops;                     // < 0: not given
};
struct Accounting {
  std::atomic<int64_t> launches{0}, host_ns{0}, host_calls{0};
  std::atomic<bool> timing{false}, clock{false};
  std::atomic<uint64_t> status_pending{0};   // bit d: kernels with bounded waits ran on device d since the last check
  std::mutex mu;
  std::vector<TimedCall> calls;
};
extern Accounting acct;

struct CallInfo {
  int64_t bytes = 0, l2_bytes = -1, edge_columns = -1;
  double flops = -1;
};
void timed_begin(const char* name, const CallInfo& info, cudaStream_t st, TimedCall& rec);
void timed_end(cudaStream_t st, TimedCall& rec);
int64_t now_ns();
[[noreturn]] void library_failure(const char* name, int rc);

// Runs `launch(stream)`, a call of the C ABI, on the current stream of the current device.
template <class F>
inline void invoke(const char* name, const CallInfo& info, F&& launch) {
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
  acct.launches.fetch_add(1, std::memory_order_relaxed);
  const bool timing = acct.timing.load(std::memory_order_relaxed), clock = acct.clock.load(std::memory_order_relaxed);
  int rc;
  if (!timing && !clock) {
    rc = launch(static_cast<void*>(st));
  } else {
    TimedCall rec{};
    const int64_t t0 = now_ns();
    if (timing) timed_begin(name, info, st, rec);
    rc = launch(static_cast<void*>(st));
    if (timing) timed_end(st, rec);
    acct.host_ns += now_ns() - t0;
    acct.host_calls += 1;
  }
  if (rc != 0) library_failure(name, rc);
}
inline void mark_status(const Tensor& t) { acct.status_pending.fetch_or(1ull << (t.get_device() & 63), std::memory_order_relaxed); }

// ---- ops ------------------------------------------------------------------------------------------
struct Packed {           // a compressed activation: quantize_activation's result without the number of bits
  Tensor codes, scale, mn;
};

Packed quantize_pack(const Tensor& x, int64_t bits, const OptTensor& noise, uint64_t seed, uint64_t offset, int64_t row_offset);
// the same with Philox noise on fp32 rows of any pitch
Packed quantize_pack_rows(const Tensor& x, int64_t bits, uint64_t seed, uint64_t offset, int64_t row_offset);
Tensor unpack(const Tensor& codes, int64_t bits, const Tensor& scale, const Tensor& mn, int64_t N, int64_t D);
Tensor rademacher(int64_t rows, int64_t cols, uint64_t seed, uint64_t offset, const Tensor& like);
bool rp_supported(int64_t D, int64_t k);
// x: rows of any pitch
Packed rp_quantize_pack(const Tensor& x, const Tensor& R, int64_t bits, uint64_t seed, uint64_t offset, int64_t row_offset,
                        Tensor* projection = nullptr);
bool linear_supported(const Tensor& a);
Tensor rows16(const Tensor& a);
// fp32 operands; w may be a transposed view (its rows are read through both strides); addend: rows of any pitch
Tensor linear(const Tensor& a, const Tensor& w, const OptTensor& bias, const OptTensor& a2, const OptTensor& w2,
              const OptTensor& out, bool accumulate, int64_t k_chunk = 0, const OptTensor& addend = {});
bool grad_weight_takes(const Tensor& g);
Tensor rows_reduce_mm(const Tensor& g, const Tensor& x, int64_t batches = 512);
Tensor grad_weight(const Tensor& g, int64_t bits, const Packed& q0, int64_t k0, const Packed* q1, int64_t k1);
std::tuple<Tensor, Tensor> rows_scale_colsum(const Tensor& g, const OptTensor& rowscale, bool want_scaled, bool want_colsum);
// (D^-1 g, g itself, both zero-padded to whole 16-byte pieces, g.sum(0))
std::tuple<Tensor, Tensor, Tensor> rows_scale_copy_colsum(const Tensor& g, const OptTensor& rowscale, bool want_colsum);
// (fp16 copy of g zero-padded to whole 16-byte pieces, g.sum(0))
std::tuple<Tensor, Tensor> rows_half_colsum(const Tensor& g, bool want_colsum);
// (y, mean, invstd); the running statistics are moved in place
std::tuple<Tensor, Tensor, Tensor> bn_forward(const Tensor& x, const OptTensor& weight, const OptTensor& bias,
                                              const OptTensor& running_mean, const OptTensor& running_var, double momentum,
                                              double eps);
// (dropout(relu(y)), its mask, mean, invstd): act_forward on bn_forward's result, without that result
std::tuple<Tensor, Tensor, Tensor, Tensor> bn_act_forward(const Tensor& x, const OptTensor& weight, const OptTensor& bias,
                                                          const OptTensor& running_mean, const OptTensor& running_var,
                                                          double momentum, double eps, double p, uint64_t seed, uint64_t offset,
                                                          int64_t index_offset);
// mask (with its p): g is the gradient of bn_act_forward's output
std::tuple<Tensor, Tensor, Tensor> bn_backward(const Tensor& g, const Packed& q, int64_t bits, const OptTensor& weight,
                                               const Tensor& mean, const Tensor& invstd, bool train, bool want_input,
                                               bool want_weight, bool want_bias, const OptTensor& mask = {}, double p = 0.0);
std::tuple<Tensor, Tensor> act_forward(int64_t op, const Tensor& x, double param, const OptTensor& uniforms, uint64_t seed,
                                       uint64_t offset, int64_t index_offset);
Tensor act_backward(int64_t op, const Tensor& g, const Tensor& mask, double param);

enum { ACT_RELU = 0, ACT_DROPOUT = 1, ACT_RELU_DROPOUT = 2, ACT_LEAKY_RELU = 3 };

// What the SpMM kernels know about the rows of a CSR structure besides the structure itself.  Each part is made when a call
// first needs it and then kept; it takes the structure's arrays as arguments so that the plan keeps neither alive.
struct RowPlan {
  // Rows with more than `threshold` edges cut into pieces (exact_spmm_split), listed by the column of their first edge:
  // pieces of different hub rows that gather the same source rows then run together.  Empty when there is no such row.
  struct Pieces {
    Tensor row, begin, end, slot, long_row, long_ptr;
    int64_t n = 0, n_long = 0;
  };
  int64_t threshold = 0;       // fp32; 0: rows are never cut
  int64_t threshold_f16 = 0;   // fp16: rows above it are chained by two warps
  const Pieces& pieces(const Tensor& rowptr, const Tensor& col) const;
  const Tensor& row_order(const Tensor& rowptr) const;     // rows by length, longest first
  int64_t n_long_f16(const Tensor& rowptr) const;          // how many of them are above threshold_f16

 private:
  mutable std::mutex mu;
  mutable std::optional<Pieces> cut;
  mutable Tensor order;
  mutable int64_t n_f16 = -1;
};
using PlanPtr = std::shared_ptr<const RowPlan>;
Tensor spmm(const Tensor& rowptr, const Tensor& col, const RowPlan& plan, const OptTensor& value, const Tensor& mat, bool mean,
            const OptTensor& bias = {});

// (best value, winning edge) of the max / min aggregation, and its gradients (grad_value, grad_mat)
std::tuple<Tensor, Tensor> spmm_minmax(const Tensor& rowptr, const Tensor& col, const RowPlan& plan, const OptTensor& value,
                                       const Tensor& mat, bool is_max);
std::tuple<Tensor, Tensor> spmm_minmax_backward(const Tensor& col, const OptTensor& value, const OptTensor& mat, const Tensor& arg,
                                                const Tensor& grad, bool need_value, bool need_mat, int64_t mat_rows);
// gradient with respect to the edge values of a sum or mean
Tensor spmm_value_backward(const Tensor& row, const Tensor& rowptr, const Tensor& col, const Tensor& mat, const Tensor& grad,
                           bool mean);

struct Csr {
  Tensor rowptr, col;
  OptTensor value;
  PlanPtr plan;
};
inline Tensor spmm(const Csr& a, const OptTensor& value, const Tensor& mat, bool mean, const OptTensor& bias = {}) {
  return spmm(a.rowptr, a.col, *a.plan, value, mat, mean, bias);
}

// (grad of mat, grad of the values) of a weighted sum or mean; t: the transpose with its weights, perm as its edges' forward
// positions, fw_rowptr: the forward rows of a mean
std::tuple<Tensor, Tensor> spmm_weighted_backward(const Csr& t, const Tensor& perm, const OptTensor& fw_rowptr, const Tensor& mat,
                                                  const Tensor& grad);

}  // namespace exb

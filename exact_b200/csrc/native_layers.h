// Autograd nodes of whole layers on a single GPU's graph (native.h has the ops they are made of).
#pragma once
#include <torch/csrc/autograd/custom_function.h>

#include "native.h"

namespace exb {

// The adjacency of a layer: forward structure, its transpose (for the dense operand's gradient) and, for a mean without
// edge values, 1 / max(row length, 1).
struct Graph : torch::CustomClassHolder {
  Csr fw, bw;
  OptTensor inv_degree;
};

// How a layer saves its activation, and the noise it draws: `offset` is the first of the call's offsets.
struct Saving {
  int64_t bits = 2, kept = 0;        // kept: columns after the random projection, 0 without one
  uint64_t seed = 0, offset = 0;
  int64_t row_offset = 0;
  bool fused = true;                 // projection and packing in one kernel where the shape allows it
};

Tensor act_node(const Tensor& x, int64_t op, double param, const OptTensor& uniforms, uint64_t seed, uint64_t offset,
                int64_t index_offset);
Tensor gcn_node(const Tensor& x, const Tensor& w, const OptTensor& b, const c10::intrusive_ptr<Graph>& graph, const Saving& how,
                bool half);
Tensor sage_node(const Tensor& x, const Tensor& w_l, const OptTensor& b_l, const OptTensor& w_r,
                 const c10::intrusive_ptr<Graph>& graph, bool mean, const Saving& how, bool projected_first,
                 bool gradient_first);
// Training batch norm with its input saved compressed (qbatch_norm, ops.py:206-254).
Tensor bn_node(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
               const OptTensor& running_var, double momentum, double eps, const Saving& how);
// The same with the ReLU and dropout (probability p, noise at `drop_offset`) that follow it.
Tensor bn_act_node(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
                   const OptTensor& running_var, double momentum, double eps, const Saving& how, double p, uint64_t drop_offset);

// reduce(A, x) with gradients to x and, when they ask for one, the edge values (qspmm_sum / mean / max / min).
// reduce: 0 sum, 1 mean, 2 max, 3 min; the graph's transpose carries the weights of the reduction.  row: the row of every edge
// (needed for the values' gradient of a sum or mean).  keep_x: the values' gradient will be asked for, x is saved compressed.
// perm: the forward position of the transpose's edges, when both gradients of a weighted sum or mean may be asked for.
Tensor aggregate_node(const Tensor& x, const OptTensor& value, const OptTensor& row, const OptTensor& perm,
                      const c10::intrusive_ptr<Graph>& graph, int64_t reduce, bool keep_x, const Saving& how);

// The same layers without anything saved (evaluation).
Tensor gcn_eval(const Tensor& x, const Tensor& w, const OptTensor& b, const c10::intrusive_ptr<Graph>& graph, bool half);
Tensor sage_eval(const Tensor& x, const Tensor& w_l, const OptTensor& b_l, const OptTensor& w_r,
                 const c10::intrusive_ptr<Graph>& graph, bool mean, bool half);

}  // namespace exb

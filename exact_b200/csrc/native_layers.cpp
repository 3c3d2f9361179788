// See native_layers.h.  Each node keeps the tensors the reference's nodes keep (ops.py:128-178, 257-371; layers.py:123-178,
// 215-265), compressed; what they are made of runs in C++ from the first check to the last launch.
#include "native_layers.h"

#include <ATen/ThreadLocalState.h>

namespace exb {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

// Library ops inside a node: no autograd bookkeeping, and no autocast (the node has cast what it casts).
struct Plain {
  at::AutoDispatchBelowADInplaceOrView below;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)};
};

template <class T>
c10::intrusive_ptr<T> state_of(AutogradContext* ctx) {
  auto it = ctx->saved_data.find("s");
  if (it == ctx->saved_data.end())
    throw std::runtime_error("the compressed activations of this layer were released by an earlier backward pass");
  auto s = c10::static_intrusive_pointer_cast<T>(it->second.toCapsule());
  ctx->saved_data.clear();   // freed when the backward is done, as `del ctx.saved` does
  return s;
}

struct Compressed {
  Packed q;
  Tensor R;            // [D, k] of a projected activation
  int64_t width = 0;   // columns of the packed activation
};

// (input2rp ->) quantize_activation (ops.py:142-149).  Uses one offset, two with a projection.
Compressed compress(const Tensor& x, const Saving& how, uint64_t offset) {
  Compressed c;
  if (how.kept == 0) {
    c.q = quantize_pack(x, how.bits, {}, how.seed, offset, how.row_offset);
    c.width = x.size(1);
    return c;
  }
  c.width = how.kept;
  c.R = rademacher(x.size(1), how.kept, how.seed, offset, x);
  if (x.scalar_type() == at::kFloat && how.fused && rp_supported(x.size(1), how.kept)) {
    c.q = rp_quantize_pack(x, c.R, how.bits, how.seed, offset + 1, how.row_offset);
    return c;
  }
  Tensor y;
  if (x.scalar_type() == at::kFloat) {
    y = linear(x, c.R.t(), {}, {}, {}, {}, false);
  } else {
    c.R = c.R.to(x.scalar_type());
    y = at::matmul(x, c.R);
  }
  c.q = quantize_pack(y, how.bits, {}, how.seed, offset + 1, how.row_offset);
  return c;
}

// g^T x_hat for a saved activation: [O, in_features].
Tensor weight_grad(const Tensor& g, const Compressed& c, int64_t bits, int64_t N) {
  Tensor G;
  if (grad_weight_takes(g)) {
    G = grad_weight(g, bits, c.q, c.width, nullptr, 0).narrow(1, 0, c.width);
  } else {
    const Tensor x = unpack(c.q.codes, bits, c.q.scale, c.q.mn, N, c.width);
    G = g.scalar_type() == at::kFloat ? rows_reduce_mm(g.contiguous(), x) : at::mm(g.t(), x);
  }
  return c.R.defined() ? at::mm(G, c.R.t()) : G.contiguous();
}

// Products by the kernel that adds sums of 64 columns up in fp32 (exact_linear_forward_strided): the gradients, evaluation, and the
// forward pass of layers that project what they save.  Without a projection the next layer quantises the product itself, whose codes
// follow its last bits, and the kernel that it always came from stays (csrc/linear_tf32.cu).
constexpr int64_t kSumChunk = 64;
int64_t forward_chunk(const Saving& how) { return how.kept ? kSumChunk : 0; }

// A (x W^T) + b with fewer columns in than out: (A x) W^T gathers the narrower operand.
bool aggregates_first(const Tensor& x, const Tensor& w) { return x.size(1) < w.size(0) && x.size(1) % 4 == 0; }

// A (x W^T) + b
Tensor gcn_product(const Graph& g, const Tensor& x, const Tensor& w, const OptTensor& b, int64_t chunk) {
  if (aggregates_first(x, w)) return linear(spmm(g.fw, g.fw.value, x, false), w, b, {}, {}, {}, false, chunk);
  return spmm(g.fw, g.fw.value, linear(x, w, {}, {}, {}, {}, false, chunk), false, b);
}

}  // namespace

// ---- activations --------------------------------------------------------------------------------------
struct ActNode : Function<ActNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t op, double param, const OptTensor& uniforms, int64_t seed,
                        int64_t offset, int64_t index_offset) {
    auto [out, mask] = act_forward(op, x, param, uniforms, (uint64_t)seed, (uint64_t)offset, index_offset);
    ctx->save_for_backward({mask});
    ctx->saved_data["op"] = op;
    ctx->saved_data["param"] = param;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Plain plain;
    Tensor g = act_backward(ctx->saved_data["op"].toInt(), grads[0], ctx->get_saved_variables()[0],
                            ctx->saved_data["param"].toDouble());
    return {g, {}, {}, {}, {}, {}, {}};
  }
};

Tensor act_node(const Tensor& x, int64_t op, double param, const OptTensor& uniforms, uint64_t seed, uint64_t offset,
                int64_t index_offset) {
  return ActNode::apply(x, op, param, uniforms, (int64_t)seed, (int64_t)offset, index_offset);
}

// ---- GCN: A (x W^T) + b ---------------------------------------------------------------------------------
struct GcnState : torch::CustomClassHolder {
  c10::intrusive_ptr<Graph> graph;
  Saving how;
  Compressed x;
  Tensor w;            // as used by the products (half under autocast)
  bool has_bias, half, x_half = false;
  int64_t rows;
};

struct GcnNode : Function<GcnNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_, const OptTensor& b,
                        const c10::intrusive_ptr<GcnState>& s) {
    const Graph& g = *s->graph;
    Tensor x = x_.contiguous(), w = w_.detach();
    Tensor out;
    if (s->half) {
      // autocast: the quantised ops cast to half (ops.py:130, 260), the products are the library's half GEMMs
      s->x_half = x.scalar_type() == at::kHalf;
      x = x.to(at::kHalf);
      w = w.to(at::kHalf);
      s->x = compress(x, s->how, s->how.offset);
      out = spmm(g.fw, g.fw.value, at::linear(x, w), false, b);   // with a bias: half + float is a float
    } else {
      s->x = compress(x, s->how, s->how.offset);
      out = gcn_product(g, x, w, b, forward_chunk(s->how));
    }
    s->w = w;
    s->rows = x.size(0);
    s->has_bias = b.has_value();
    ctx->saved_data["s"] = c10::IValue::make_capsule(s);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Plain plain;
    auto s = state_of<GcnState>(ctx);
    const Graph& gr = *s->graph;
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    Tensor g = grads[0].contiguous(), gb, gw, gx;
    const int64_t O = g.size(1);
    if (s->half) {
      Tensor g16 = g;      // without a bias the output, and so its gradient, is half
      if (g.scalar_type() == at::kFloat) {
        auto [h, sum] = rows_half_colsum(g, s->has_bias);
        g16 = h;           // padded with zero columns to whole 16-byte pieces
        gb = sum;
      }
      if (need_x || need_w) {
        const Tensor gh = spmm(gr.bw, gr.bw.value, g16, false).narrow(1, 0, O);
        if (need_w) gw = weight_grad(gh, s->x, s->how.bits, s->rows).to(at::kFloat);
        if (need_x) gx = s->x_half ? at::mm(gh, s->w) : at::mm(gh, s->w, at::kFloat);
      }
      return {gx, gw, gb, {}};
    }
    if (O % 4) {
      // whole 16-byte column groups for the gather, the bias gradient on the way
      auto [padded, sum] = rows_scale_colsum(g, {}, true, s->has_bias);
      g = padded;
      gb = sum;
    } else if (s->has_bias) {
      gb = std::get<1>(rows_scale_colsum(g, {}, false, true));
    }
    if (need_x || need_w) {
      const Tensor gh = spmm(gr.bw, gr.bw.value, g, false);
      if (need_w) {
        gw = weight_grad(gh, s->x, s->how.bits, s->rows);
        if (O % 4) gw = gw.narrow(0, 0, O);
      }
      if (need_x) gx = linear(gh.narrow(1, 0, O), s->w.t(), {}, {}, {}, {}, false, kSumChunk);
    }
    return {gx, gw, gb, {}};
  }
};

Tensor gcn_node(const Tensor& x, const Tensor& w, const OptTensor& b, const c10::intrusive_ptr<Graph>& graph, const Saving& how,
                bool half) {
  auto s = c10::make_intrusive<GcnState>();
  s->graph = graph;
  s->how = how;
  s->half = half;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)};
  return GcnNode::apply(x, w, b, s);
}

// ---- GraphSAGE: reduce(A, x) W_l^T + b (+ x W_r^T) -------------------------------------------------------
// The compressed tensors are those of the reference's nodes (x once, shared by the aggregation and lin_r; reduce(A, x) for
// lin_l), drawn in the same order; results differ by fp32 reassociation only.
struct SageState : torch::CustomClassHolder {
  c10::intrusive_ptr<Graph> graph;
  Saving how;
  Compressed x, agg;
  Tensor w_l, w_r;
  bool mean, has_bias, gradient_first, projected_first;
  int64_t rows;
};

struct SageNode : Function<SageNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_l_, const OptTensor& b, const OptTensor& w_r_,
                        const c10::intrusive_ptr<SageState>& s) {
    const Graph& g = *s->graph;
    Tensor x = x_.contiguous();
    const Tensor w_l = w_l_.detach();
    const int64_t out_f = w_l.size(0), in_f = w_l.size(1);
    OptTensor w_r;
    if (w_r_) w_r = w_r_->detach();
    s->w_l = w_l;
    if (w_r) s->w_r = *w_r;
    s->rows = x.size(0);
    s->has_bias = b.has_value();
    uint64_t offset = s->how.offset;
    const Tensor rows = rows16(x);            // several products read them, the projection among them
    if (w_r) s->x = compress(s->how.kept ? rows : x, s->how, offset);
    offset += s->how.kept ? 2 : 1;            // without lin_r nothing reads it; the noise stays that of the separate nodes
    x = rows;
    const int64_t k = s->how.kept, kp = (k + 3) / 4 * 4, op = (out_f + 3) / 4 * 4;
    Tensor out;
    if (s->projected_first && k && kp + op < in_f) {
      // Few outputs: reduce(A, x) R = reduce(A, x R) and reduce(A, x) W_l^T = reduce(A, x W_l^T), so the SpMM works on
      // k + out_features columns and its result holds what lin_l saves (ops.py:142-149) and lin_l's output.
      s->agg.R = rademacher(in_f, k, s->how.seed, offset, x);
      s->agg.width = k;
      Tensor wcat = at::zeros({kp + op, in_f}, w_l.options());
      wcat.narrow(0, 0, k).copy_(s->agg.R.t());
      wcat.narrow(0, kp, out_f).copy_(w_l);
      const Tensor t = spmm(g.fw, g.fw.value, linear(x, wcat, {}, {}, {}, {}, false, forward_chunk(s->how)), s->mean);
      s->agg.q = quantize_pack_rows(t.narrow(1, 0, k), s->how.bits, s->how.seed, offset + 1, s->how.row_offset);
      const Tensor part = t.narrow(1, kp, out_f);
      if (w_r) out = linear(x, *w_r, b, {}, {}, {}, false, forward_chunk(s->how), part);
      else out = b ? part.add(*b) : part.contiguous();
    } else {
      const Tensor agg = spmm(g.fw, g.fw.value, x, s->mean);
      s->agg = compress(agg, s->how, offset);
      OptTensor a2;
      if (w_r) a2 = x;
      out = linear(agg, w_l, b, a2, w_r, {}, false, forward_chunk(s->how));
    }
    ctx->saved_data["s"] = c10::IValue::make_capsule(s);
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Plain plain;
    auto s = state_of<SageState>(ctx);
    const Graph& gr = *s->graph;
    const bool need_x = ctx->needs_input_grad(0), has_r = s->w_r.defined();
    Tensor g = grads[0].contiguous(), gx, gl, gb, gwr;
    const int64_t O = g.size(1), in_f = s->w_l.size(1), k = s->agg.width;
    const bool aggregate_g = need_x && s->gradient_first && O <= in_f;
    const bool by_degree = s->mean && gr.inv_degree.has_value();
    // One pass over g: D^-1 g, the operand of the transposed mean, g with its rows padded to whole 16-byte pieces for the
    // products below, and the bias gradient g.sum(0) (backward_func.cc:88-90).
    Tensor scaled;
    if (aggregate_g && by_degree && O % 4) {
      auto [sc, padded, sum] = rows_scale_copy_colsum(g, gr.inv_degree, s->has_bias);
      scaled = sc;
      g = padded;
      gb = sum;
    } else if (O % 4 || (aggregate_g && by_degree)) {
      auto [sc, sum] = rows_scale_colsum(g, O % 4 ? OptTensor() : gr.inv_degree, true, s->has_bias);
      (O % 4 ? g : scaled) = sc;
      gb = sum;
    } else if (s->has_bias) {
      gb = std::get<1>(rows_scale_colsum(g, {}, false, true));
    }
    // both weight gradients in one pass over g: g^T [Xq_agg | Xq_x], then the two small transposed projections
    if (grad_weight_takes(g)) {
      const int64_t k0pad = (k + 15) / 16 * 16;
      const Tensor G = grad_weight(g, s->how.bits, s->agg.q, k, has_r ? &s->x.q : nullptr, has_r ? s->x.width : 0).narrow(0, 0, O);
      gl = G.narrow(1, 0, k);
      if (has_r) gwr = G.narrow(1, k0pad, s->x.width);
      gl = s->agg.R.defined() ? at::mm(gl, s->agg.R.t()) : gl.contiguous();
      if (has_r) gwr = s->x.R.defined() ? at::mm(gwr, s->x.R.t()) : gwr.contiguous();
    } else {
      gl = weight_grad(g, s->agg, s->how.bits, s->rows).narrow(0, 0, O);
      if (has_r) gwr = weight_grad(g, s->x, s->how.bits, s->rows).narrow(0, 0, O);
    }
    if (need_x) {
      const Tensor g_true = g.narrow(1, 0, O);
      OptTensor a2, w2;
      if (has_r) {
        a2 = g_true;
        w2 = s->w_r.t();
      }
      if (aggregate_g) {
        // A^T (D^-1 g) reads no edge weights; with edge values, or a sum, the transposed structure's weights apply
        const Tensor t = spmm(gr.bw, by_degree ? OptTensor() : gr.bw.value, scaled.defined() ? scaled : g, false);
        gx = linear(t.narrow(1, 0, O), s->w_l.t(), {}, a2, w2, {}, false, kSumChunk);
      } else {
        Tensor y = linear(g_true, s->w_l.t(), {}, {}, {}, {}, false, kSumChunk);
        if (by_degree) y.mul_(gr.inv_degree->unsqueeze(1));   // the transposed structure carries no weights of the mean
        gx = spmm(gr.bw, gr.bw.value, y, false);
        if (has_r) linear(g_true, s->w_r.t(), {}, {}, {}, gx, true, kSumChunk);
      }
    }
    return {gx, gl, gb, gwr, {}};
  }
};

Tensor sage_node(const Tensor& x, const Tensor& w_l, const OptTensor& b_l, const OptTensor& w_r,
                 const c10::intrusive_ptr<Graph>& graph, bool mean, const Saving& how, bool projected_first,
                 bool gradient_first) {
  auto s = c10::make_intrusive<SageState>();
  s->graph = graph;
  s->how = how;
  s->mean = mean;
  s->projected_first = projected_first;
  s->gradient_first = gradient_first;
  return SageNode::apply(x, w_l, b_l, w_r, s);
}

// ---- batch norm: qbatch_norm (ops.py:206-254) ---------------------------------------------------------------
struct BnState : torch::CustomClassHolder {
  Packed x;
  Tensor mean, invstd;
  OptTensor weight;
  int64_t bits;
  bool act = false;              // ReLU and dropout follow
  double p = 0.0;
  uint64_t drop_offset = 0;
};

struct BnNode : Function<BnNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const OptTensor& weight, const OptTensor& bias,
                        const OptTensor& running_mean, const OptTensor& running_var, double momentum, double eps,
                        const c10::intrusive_ptr<BnState>& s, const Saving& how) {
    const Tensor x = x_.contiguous();
    s->x = quantize_pack(x, how.bits, {}, how.seed, how.offset, how.row_offset);
    Tensor y;
    if (s->act) {
      Tensor mask;
      std::tie(y, mask, s->mean, s->invstd) =
          bn_act_forward(x, weight, bias, running_mean, running_var, momentum, eps, s->p, how.seed, s->drop_offset,
                         how.row_offset * x.size(1));
      ctx->save_for_backward({mask});
    } else {
      std::tie(y, s->mean, s->invstd) = bn_forward(x, weight, bias, running_mean, running_var, momentum, eps);
    }
    if (weight) s->weight = weight->detach();
    s->bits = how.bits;
    ctx->saved_data["s"] = c10::IValue::make_capsule(s);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Plain plain;
    auto s = state_of<BnState>(ctx);
    OptTensor mask;
    if (s->act) mask = ctx->get_saved_variables()[0];
    auto [gx, gw, gb] = bn_backward(grads[0], s->x, s->bits, s->weight, s->mean, s->invstd, true, ctx->needs_input_grad(0),
                                    s->weight && ctx->needs_input_grad(1), s->weight && ctx->needs_input_grad(2), mask, s->p);
    return {gx, gw, gb, {}, {}, {}, {}, {}, {}};
  }
};

Tensor bn_node(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
               const OptTensor& running_var, double momentum, double eps, const Saving& how) {
  return BnNode::apply(x, weight, bias, running_mean, running_var, momentum, eps, c10::make_intrusive<BnState>(), how);
}

Tensor bn_act_node(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
                   const OptTensor& running_var, double momentum, double eps, const Saving& how, double p, uint64_t drop_offset) {
  auto s = c10::make_intrusive<BnState>();
  s->act = true;
  s->p = p;
  s->drop_offset = drop_offset;
  return BnNode::apply(x, weight, bias, running_mean, running_var, momentum, eps, s, how);
}

// ---- aggregation: qspmm_sum / mean / max / min (ops.py:257-436) --------------------------------------------
struct AggregateState : torch::CustomClassHolder {
  c10::intrusive_ptr<Graph> graph;
  Saving how;
  OptTensor value, row, perm;
  Compressed x;        // only when the edge values get a gradient: nothing else reads it
  Tensor arg;
  int64_t reduce, rows;
  bool keep_x;
};

// Whether both gradients of a weighted sum or mean come from one walk (exact_spmm_weighted_backward, up to 256 columns).  It gives
// a row of the transpose a warp, of which few columns use few lanes, where the separate kernels take several short rows, or 32
// edges, a warp.  So many rows of few edges and columns stay with those: below (56 - columns) / 5 edges a row, from 65,536 rows on
// (one to three columns, whose rows are no whole 16-byte pieces: from 2^20).  With long rows, whose pieces the separate kernels wait
// for twice, from 2^18 rows on, and up to 2^20 at half as many edges.  Both gradients, one walk over separate, random graphs of
// 3 | 7 | 11 | 21 edges a row:
//     columns      4                          16                         24                    32                    64
//     40,000       1.09 | 0.96 | 0.79         1.00 | 0.94 | 0.79         0.97 | 0.92 | 0.79    0.94 | 0.93 | 0.86    0.88 | 0.89 | 0.80
//     170,000      1.58 | 1.16 | 0.96 | 0.75  1.50 | 1.09 | 0.93 | 0.74  1.21 | 0.99 | 0.86    1.14 | 0.94 | 0.82    0.95 | 0.88 | 0.80
//     500,000      1.86 | 1.26 | 1.00 | 0.77  1.49 | 1.18 | 0.98 | 0.81  1.32 | 1.08 | 0.93    1.19 | 0.97 | 0.85    1.01 | 0.84 | 0.75
//     2,000,000    2.12 | 1.43                1.55 | 1.10                1.33 | 1.01           1.25 | 0.97           1.04 | 0.86
//     power-law graphs: 170,000 at most 0.98 anywhere, 500,000 with 4 and 16 columns 1.29 | 1.05 | 0.92 and 1.09 | 0.89 | 0.85,
//     2,000,000 of 3 | 7 edges 1.98 | 1.33 and 1.45 | 1.08.
// What the lines leave: 1.22 for two columns of 500,000 x 7, 1.13 at worst elsewhere.
bool one_walk(const Graph& g, int64_t K, int64_t nnz) {
  if (K > 256 || nnz == 0) return false;
  const int64_t M = g.bw.rowptr.size(0) - 1;
  if (M < (1 << 16) || 5 * nnz >= (56 - K) * M) return true;
  if (g.bw.plan->pieces(g.bw.rowptr, g.bw.col).n * 4096 > M && M < (1 << 20)) return M < (1 << 18) || K < 4 || 10 * nnz >= (56 - K) * M;
  return K < 4 && M < (1 << 20);
}

struct AggregateNode : Function<AggregateNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const OptTensor& value, const c10::intrusive_ptr<AggregateState>& s) {
    const Graph& g = *s->graph;
    const Tensor x = x_.contiguous();
    Tensor out;
    if (s->reduce <= 1) {
      out = spmm(g.fw, value, x, s->reduce == 1);
    } else {
      auto [best, arg] = spmm_minmax(g.fw.rowptr, g.fw.col, *g.fw.plan, value, x, s->reduce == 2);
      out = best;
      s->arg = arg;
    }
    if (s->keep_x) s->x = compress(x, s->how, s->how.offset);
    if (value) s->value = value->detach();
    s->rows = x.size(0);
    ctx->saved_data["s"] = c10::IValue::make_capsule(s);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Plain plain;
    auto s = state_of<AggregateState>(ctx);
    const Graph& gr = *s->graph;
    const bool need_x = ctx->needs_input_grad(0), need_v = s->value && ctx->needs_input_grad(1);
    const Tensor g = grads[0].contiguous();
    Tensor gx, gv, x;
    if (need_v) {
      x = unpack(s->x.q.codes, s->how.bits, s->x.q.scale, s->x.q.mn, s->rows, s->x.width);
      if (s->x.R.defined()) x = linear_supported(x) ? linear(x, s->x.R, {}, {}, {}, {}, false) : at::matmul(x, s->x.R.t());
    }
    if (s->reduce <= 1 && need_v && need_x && s->perm && gr.bw.value && one_walk(gr, g.size(1), gr.fw.col.size(0))) {
      OptTensor rows;
      if (s->reduce == 1) rows = gr.fw.rowptr;
      std::tie(gx, gv) = spmm_weighted_backward(gr.bw, *s->perm, rows, x, g);
    } else if (s->reduce <= 1) {
      if (need_v) gv = spmm_value_backward(*s->row, gr.fw.rowptr, gr.fw.col, x, g, s->reduce == 1);
      if (need_x) gx = spmm(gr.bw, gr.bw.value, g, false);
    } else {
      OptTensor mat;
      if (need_v) mat = x;
      auto [v, m] = spmm_minmax_backward(gr.fw.col, s->value, mat, s->arg, g, need_v, need_x, s->rows);
      gv = v;
      gx = m;
    }
    return {gx, gv, {}};
  }
};

Tensor aggregate_node(const Tensor& x, const OptTensor& value, const OptTensor& row, const OptTensor& perm,
                      const c10::intrusive_ptr<Graph>& graph, int64_t reduce, bool keep_x, const Saving& how) {
  auto s = c10::make_intrusive<AggregateState>();
  s->keep_x = keep_x;
  s->graph = graph;
  s->how = how;
  s->row = row;
  s->perm = perm;
  s->reduce = reduce;
  return AggregateNode::apply(x, value, s);
}

// ---- evaluation -----------------------------------------------------------------------------------------
// Evaluation is compared with the plain fp32 model, so its products are no further from the exact ones than the library's fp32 GEMM:
// 1.06e-7 to 1.2e-7 (Frobenius) from 100 columns on against 1.8e-7 at 100, 2.0e-7 at 256 and 4.4e-7 at 602.  (Where one feature outweighs
// the others: 1.1e-7 .. 1.35e-7 against 1.0e-7 .. 1.3e-7, sums of few terms round less.)  Up to 64 columns the
// library is the nearer one (9e-8 against 1.04e-7 at 48) and takes them, 200,000 x 48 -> 256 in 173 us against 58.
constexpr int64_t kEvalLibrary = 64;

// a w^T (+ a2 w2^T) (+ bias) (+ addend)
Tensor eval_product(const Tensor& a, const Tensor& w, const OptTensor& bias = {}, const OptTensor& a2 = {}, const OptTensor& w2 = {},
                    const OptTensor& addend = {}) {
  if (a.size(1) + (a2 ? a2->size(1) : 0) > kEvalLibrary) return linear(a, w, bias, a2, w2, {}, false, kSumChunk, addend);
  Tensor out = at::linear(a, w, bias);
  if (a2) out.addmm_(*a2, w2->t());
  return addend ? out.add_(*addend) : out;
}

Tensor gcn_eval(const Tensor& x_, const Tensor& w, const OptTensor& b, const c10::intrusive_ptr<Graph>& graph, bool half) {
  Plain plain;
  const Graph& g = *graph;
  if (!half) {
    const Tensor x = x_.contiguous();
    if (aggregates_first(x, w)) return eval_product(spmm(g.fw, g.fw.value, x, false), w, b);
    return spmm(g.fw, g.fw.value, eval_product(x, w), false, b);
  }
  return spmm(g.fw, g.fw.value, at::linear(x_.to(at::kHalf), w.to(at::kHalf)), false, b);
}

Tensor sage_eval(const Tensor& x_, const Tensor& w_l, const OptTensor& b, const OptTensor& w_r,
                 const c10::intrusive_ptr<Graph>& graph, bool mean, bool half) {
  Plain plain;
  const Graph& g = *graph;
  if (half) {
    const Tensor x = x_.to(at::kHalf).contiguous();
    OptTensor b16;
    if (b) b16 = b->to(at::kHalf);
    Tensor out = at::linear(spmm(g.fw, g.fw.value, x, mean), w_l.to(at::kHalf), b16);
    return w_r ? out.add_(at::linear(x, w_r->to(at::kHalf))) : out;
  }
  const int64_t out_f = w_l.size(0), in_f = w_l.size(1), pad = (4 - out_f % 4) % 4;
  const Tensor x = x_.contiguous();
  if (out_f + pad >= in_f) {
    const Tensor agg = spmm(g.fw, g.fw.value, x, mean);
    OptTensor a2;
    if (w_r) a2 = x;
    return eval_product(agg, w_l, b, a2, w_r);
  }
  // fewer outputs than inputs: reduce(A, x) W_l^T = reduce(A, x W_l^T) gathers the narrower operand
  const Tensor rows = rows16(x);
  const Tensor t = spmm(g.fw, g.fw.value, eval_product(rows, pad ? at::constant_pad_nd(w_l, {0, 0, 0, pad}) : w_l), mean);
  const Tensor part = t.narrow(1, 0, out_f);
  if (w_r) return eval_product(rows, *w_r, b, {}, {}, part);
  return b ? part.add(*b) : part.contiguous();
}

}  // namespace exb

"""Stand-in for the reference's `exact.cpp_extension.backward_func` module
(exact/exact/cpp_extension/backward_func.cc:83-107): the dense-layer GEMMs and ATen batch-norm
pass-throughs.  The tall GEMMs (rows = nodes) go to the tensor-core kernel with fp32-equivalent accuracy
(exact_linear_forward), the weight gradients to exact_grad_weight_from_packed; unsupported shapes stay library GEMMs."""
import torch

from .. import _lib
from ..conf import config


def _tc_ok(a):
    return (config.linear_tensor_core and a.is_cuda and a.dtype == torch.float32 and a.dim() == 2
            and a.size(0) >= 1024)


def _rows16(a):
    """`a` with 16-byte aligned rows: itself when its pitch already is, else a zero-padded copy."""
    if a.stride(1) == 1 and a.stride(0) % 4 == 0 and a.stride(0) >= a.size(1) and a.data_ptr() % 16 == 0:
        return a
    K = a.size(1)
    out = a.new_zeros((a.size(0), (K + 3) // 4 * 4))
    out[:, :K].copy_(a)
    return out[:, :K]


SUM_CHUNK = 64   # sums of 64 columns added in fp32: the gradients' products (exact_linear_forward_strided)


def forward_chunk():
    """How the layers' forward products are summed: as the C++ nodes do it (forward_chunk, csrc/native_layers.cpp)."""
    return SUM_CHUNK if config.kept_frac < 1.0 else 0


def linear_forward(a, weight, bias=None, a2=None, weight2=None, out=None, accumulate=False, k_chunk=0):
    """a @ weight.T (+ a2 @ weight2.T) (+ bias), optionally added to `out`: F.linear of ops.py:150 and the
    g W product of backward_func.cc:86 (pass weight.t()).  fp32 in and out."""
    if not _tc_ok(a) or (a2 is not None and not _tc_ok(a2)):
        _lib.note_library_call("F.linear (rows < 1024, not fp32 or not CUDA)")
        r = torch.nn.functional.linear(a, weight, bias)
        if a2 is not None:
            r = r.addmm_(a2, weight2.t())
        if out is not None:
            return out.add_(r) if accumulate else out.copy_(r)
        return r
    out = _lib.native().linear(a, weight, bias, a2, weight2, out, accumulate, k_chunk)
    if config.check_device_status:
        _lib.check_status(a.device, force=True)
    return out


def rows_reduce_mm(g, x, batches=512):
    """g^T x for g [M, out], x [M, k] with M in the millions and out, k small: the reduction over rows is
    cut into `batches` independent products that one batched library GEMM computes in parallel and a sum
    joins (a single GEMM call leaves most SMs idle on this shape: 2.0 ms against 0.76 ms at
    2.45M x 256 x 32).  Same fp32 arithmetic, pairwise-style summation."""
    M = g.size(0)
    _lib.note_library_call("g^T x on the unpacked activation (library GEMM)")
    if not (g.is_cuda and g.dim() == 2 and M >= 64 * batches and g.is_contiguous() and x.is_contiguous()):
        return g.t().mm(x)
    rows = M // batches * batches
    out = torch.bmm(g[:rows].view(batches, -1, g.size(1)).transpose(1, 2), x[:rows].view(batches, -1, x.size(1))).sum(0)
    if rows < M:
        out.addmm_(g[rows:].t(), x[rows:])
    return out


def grad_weight_supported(g, k0, k1, bits):
    """The shapes at which the product needs the fewest reads of g: fp32 g [N, O] with O <= 256 (padded to a multiple of 4), at
    least 4,096 rows, few activation columns.  Kept for callers that choose by it; the layers take the kernel for every
    shape of grad_weight_takes."""
    if not (config.grad_weight_tensor_core and g.is_cuda and g.dtype == torch.float32 and g.dim() == 2):
        return False
    N, O = g.shape
    kpad = (k0 + 15) // 16 * 16 + ((k1 + 15) // 16 * 16 if k1 else 0)
    # a width that is not a multiple of 4 (47 classes) goes in as a zero-padded copy of g
    return (N >= 4096 and (O + 3) // 4 * 4 <= 256 and kpad <= 256 and (k0 + k1) * (32 // (8 // bits)) <= 1024
            and g.is_contiguous() and (g.data_ptr() % 16 == 0 or O % 4 != 0))


def grad_weight_takes(g):
    """Whether the layers' weight gradients come from exact_grad_weight_from_packed: fp32 g [N, O], O <= 256, on the GPU.  The rule
    is the C++ nodes' own, so a switch that sends a layer through the Python nodes does not change the route."""
    return config.grad_weight_tensor_core and g.is_cuda and _lib.native().grad_weight_takes(g)


def grad_weight_from_packed(g, q0, k0, q1=None, k1=0):
    """(g^T Xq0 [O, k0], g^T Xq1 [O, k1] or None) for packed activations q = (packed, bits, scale_bf16, min_bf16)
    of N rows: backward_func.cc:87 with the dequantisation of ops.py:164 folded in, one pass over g."""
    q1 = (None, None, None, None) if q1 is None else q1
    k1 = k1 if q1[0] is not None else 0
    out = _lib.native().grad_weight(g, q0[1], q0[0], q0[2], q0[3], k0, q1[0], q1[2], q1[3], k1)
    if config.check_device_status:
        _lib.check_status(g.device, force=True)
    k0pad = (k0 + 15) // 16 * 16
    return out[:, :k0], (out[:, k0pad:k0pad + k1] if k1 else None)


def linear_backward(grad_output, input, weight, bias=None, need_grad_input=True):
    """backward_func.cc:83-93.  The input gradient is left out (None) when the caller has no use for it."""
    grad_input = linear_forward(grad_output, weight.t(), k_chunk=SUM_CHUNK) if need_grad_input else None
    grad_weight = rows_reduce_mm(grad_output, input)
    grad_bias = rows_scale_colsum(grad_output)[1] if bias is not None else None
    return grad_input, grad_weight, grad_bias


def native_batch_norm(input, weight, bias, running_mean, running_var, training, momentum, eps):
    return torch.ops.aten.native_batch_norm(input, weight, bias, running_mean, running_var, training, momentum, eps)


def _batch_norm_impl_index(input, weight, bias, running_mean, running_var, training, momentum, eps, cudnn_enabled):
    return torch.ops.aten._batch_norm_impl_index(input, weight, bias, running_mean, running_var, training,
                                                 momentum, eps, cudnn_enabled)


def native_batch_norm_backward(grad_out, input, weight, running_mean, running_var, save_mean, save_invstd,
                               train, eps, output_mask):
    return torch.ops.aten.native_batch_norm_backward(grad_out, input, weight, running_mean, running_var,
                                                     save_mean, save_invstd, train, eps, output_mask)


def batch_norm_backward_from_packed_supported(grad_out, quantized):
    """Whether native_batch_norm_backward can read the saved input in its packed form (this library's kernels):
    a compressed [N, D] fp32 activation with bf16 row statistics and D a multiple of 4."""
    q_input, q_bits, q_scale, q_min = quantized
    return (q_bits is not None and grad_out.is_cuda and grad_out.dtype == torch.float32 and grad_out.dim() == 2
            and grad_out.size(1) % 4 == 0 and q_scale.dtype == torch.bfloat16 and q_input.is_cuda)


def batch_norm_backward_from_packed(grad_out, quantized, weight, running_mean, running_var, save_mean, save_invstd,
                                    train, eps, output_mask):
    """native_batch_norm_backward (the call of ops.py:248-251) with the dequantisation of ops.py:238 folded into
    both of its passes: the column sums and the element-wise pass read the packed bytes and the bf16 row
    statistics, the [N, D] reconstruction is never written.  Returns (grad_input, grad_weight, grad_bias)."""
    q_input, q_bits, q_scale, q_min = quantized
    if train:
        mean, invstd = save_mean, save_invstd
    else:
        mean, invstd = running_mean, torch.rsqrt(running_var + eps)
    return _lib.native().bn_backward(grad_out, q_input, q_scale, q_min, q_bits, weight, mean, invstd, train, *output_mask)


def rows_scale_colsum(g, rowscale=None, want_scaled=False, want_colsum=True, pad_to=4):
    """One pass over g [N, K] -> (g * rowscale[:, None] zero-padded to a multiple of `pad_to` columns or None,
    g.sum(0) or None): the operand D^-1 g of the transposed mean aggregation (spmm.cc:128-137) and the bias gradient
    (backward_func.cc:88-90).  Small or non-fp32 inputs take the framework's ops."""
    N, K = g.shape
    if not (g.is_cuda and g.dtype == torch.float32 and g.dim() == 2 and g.stride(1) == 1 and N >= 1024 and pad_to == 4):
        scaled = None
        if want_scaled:
            scaled = g.new_zeros((N, (K + pad_to - 1) // pad_to * pad_to))
            scaled[:, :K] = g if rowscale is None else g * rowscale.unsqueeze(1)
        return scaled, (g.sum(0) if want_colsum else None)
    if rowscale is not None:
        rowscale = rowscale.to(torch.float32).contiguous()
    return _lib.native().rows_scale_colsum(g, rowscale, want_scaled, want_colsum)

"""Quantised nn.Modules with the reference's names and constructor arguments
(exact/exact/layers.py).  torch_geometric is not a dependency: GCNConv and SAGEConv below restate the
parts of PyG 1.7.2's layers that the reference's subclasses and QModule rely on (attributes read at
module.py:41-56, parameter shapes, initialisation, forward on a SparseTensor adjacency)."""
import math

import torch
import torch.nn.functional as F
from torch import Tensor
from torch.nn import Parameter

from . import _lib
from .conf import config
from .cpp_extension import quantization as ext_quantization
from .ops import project_and_quantize, qbatch_norm, qlinear
from .qscheme import QScheme
from .sparse import SparseTensor, gcn_norm
from .spmm import QMatmul, qmatmul, qsage_layer, sage_layer_applies


def _glorot(t):
    if t is not None:
        stdv = math.sqrt(6.0 / (t.size(-2) + t.size(-1)))
        t.data.uniform_(-stdv, stdv)


# ----------------------------------------------------------------------------------------------------
# Plain (uncompressed) layers: what a model is written with before QModule converts it.
class GCNConv(torch.nn.Module):
    """torch_geometric.nn.GCNConv (1.7.2) on a SparseTensor adjacency: out = A_hat (x W) + b."""

    def __init__(self, in_channels, out_channels, improved=False, cached=False, add_self_loops=True,
                 normalize=True, bias=True, aggr="add"):
        super().__init__()
        self.in_channels, self.out_channels = in_channels, out_channels
        self.improved, self.cached = improved, cached
        self.add_self_loops, self.normalize, self.aggr = add_self_loops, normalize, aggr
        self._cached_adj_t = None
        self.weight = Parameter(torch.empty(in_channels, out_channels))
        if bias:
            self.bias = Parameter(torch.empty(out_channels))
        else:
            self.register_parameter("bias", None)
        self.reset_parameters()

    def reset_parameters(self):
        _glorot(self.weight)
        if self.bias is not None:
            self.bias.data.zero_()
        self._cached_adj_t = None

    def _norm(self, adj_t):
        if not self.normalize:
            return adj_t
        if self._cached_adj_t is not None:
            return self._cached_adj_t
        out = gcn_norm(adj_t, add_self_loops=self.add_self_loops)
        if self.cached:
            self._cached_adj_t = out
        return out

    def forward(self, x, adj_t, edge_weight=None):
        adj_t = self._norm(adj_t)
        x = x @ self.weight
        out = qmatmul_plain(adj_t, x, "sum")
        if self.bias is not None:
            out = out + self.bias
        return out


class SAGEConv(torch.nn.Module):
    """torch_geometric.nn.SAGEConv (1.7.2), mean aggregation: out = W_l mean_j(x_j) + W_r x."""

    def __init__(self, in_channels, out_channels, normalize=False, root_weight=True, bias=True):
        super().__init__()
        self.in_channels, self.out_channels = in_channels, out_channels
        self.normalize, self.root_weight = normalize, root_weight
        self.aggr = "mean"
        if isinstance(in_channels, int):
            in_channels = (in_channels, in_channels)
        self.lin_l = torch.nn.Linear(in_channels[0], out_channels, bias=bias)
        if root_weight:
            self.lin_r = torch.nn.Linear(in_channels[1], out_channels, bias=False)
        self.reset_parameters()

    def reset_parameters(self):
        self.lin_l.reset_parameters()
        if self.root_weight:
            self.lin_r.reset_parameters()

    def forward(self, x, adj_t, size=None):
        if isinstance(x, Tensor):
            x = (x, x)
        out = qmatmul_plain(adj_t, x[0], "mean")
        out = self.lin_l(out)
        if self.root_weight and x[1] is not None:
            out = out + self.lin_r(x[1])
        if self.normalize:
            out = F.normalize(out, p=2.0, dim=-1)
        return out


def qmatmul_plain(adj_t, x, reduce):
    """Aggregation of the unconverted layers: the same SpMM kernel, nothing saved compressed."""
    saved = config.compress_activation, config.kept_frac
    config.compress_activation, config.kept_frac = False, 1.0
    try:
        return qmatmul(adj_t, x, reduce)
    finally:
        config.compress_activation, config.kept_frac = saved


# ----------------------------------------------------------------------------------------------------
class QLinear(torch.nn.Linear):
    """layers.py:268-281."""

    def __init__(self, input_features, output_features, bias=True, rp=True):
        super().__init__(input_features, output_features, bias)
        self.scheme = QScheme("linear") if config.single_precision else None
        self.rp = rp

    def forward(self, input, quantized=None, randmat=None):
        if self.training:
            return qlinear.apply(input, self.weight, self.bias, quantized, randmat, self.scheme, self.rp)
        return super().forward(input)


class QReLU(torch.nn.Module):
    """layers.py:284-292."""

    def __init__(self, inplace=False):
        super().__init__()

    def forward(self, input):
        if self.training:
            return ext_quantization.act_quantized_relu(input.contiguous())
        return F.relu(input)


class QLeakyReLU(torch.nn.Module):
    """layers.py:295-301 (the reference applies the masked kernel in training and in evaluation alike)."""

    def __init__(self, negative_slope, inplace=False):
        super().__init__()
        self.negative_slope = negative_slope

    def forward(self, input):
        return ext_quantization.act_quantized_leaky_relu(input, self.negative_slope)


class QDropout(torch.nn.Module):
    """layers.py:316-325."""

    def __init__(self, p):
        self.p = p
        super().__init__()

    def forward(self, input):
        if self.training:
            return ext_quantization.act_quantized_dropout(input.contiguous(), self.p, self.training)
        return F.dropout(input, self.p, self.training)


class ActDropout(torch.nn.Module):
    """activation followed by dropout, as the GCN / GraphSAGE models apply them after every hidden layer
    (mem_speed_bench/models/gcn.py:60-61, sage.py:72-73).  Kept as one child so that QModule can swap the
    pair for the one-pass QReLUDropout; unconverted it just calls the two modules."""

    def __init__(self, activation, dropout):
        super().__init__()
        self.activation, self.dropout = activation, dropout

    def forward(self, input):
        return self.dropout(self.activation(input))


class QReLUDropout(torch.nn.Module):
    """QReLU followed by QDropout (layers.py:284-292, 316-325) in one pass over the activation and with one
    saved 1-bit mask; outputs and gradients are those of the two modules."""

    def __init__(self, p):
        super().__init__()
        self.p = p

    def forward(self, input):
        if self.training:
            return ext_quantization.act_quantized_relu_dropout(input, self.p, True)
        return F.relu(input)


def _watched(module):
    """Whether a call of the module does anything but run the forward that its class has here: hooks, a forward replaced on the
    instance or the class (offloading and profiling wrappers), a compiled call, a replaced Module.__call__ (tracers)."""
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks
                or torch.nn.modules.module._has_any_global_hook()
                or getattr(module.forward, "__func__", None) is not _FORWARDS[type(module)]
                or getattr(module, "_compiled_call_impl", None) is not None or type(module).__call__ is not _MODULE_CALL)


def norm_act(norm, act, input):
    """act(norm(input)).  A quantised batch norm followed by QReLUDropout runs as one node, without the pass over the values in
    between, which nothing else reads; a module that is hooked or replaced is called by itself."""
    if norm is None:
        return act(input)
    if (type(norm) is QBatchNorm1d and type(act) is QReLUDropout and not _watched(norm) and not _watched(act)
            and act.training and norm.takes_activation(input)):
        return norm._normalise(input, act.p)
    return act(norm(input))


class QDropout2(torch.nn.Module):
    """layers.py:328-337."""

    def __init__(self, p):
        self.p = p
        super().__init__()

    def forward(self, input):
        if self.training:
            return ext_quantization.act_quantized_dropout(input.contiguous(), self.p, self.training) * (1 - self.p)
        return F.dropout(input, self.p, self.training) * (1 - self.p)


class QBatchNorm1d(torch.nn.BatchNorm1d):
    """layers.py:340-388."""

    def __init__(self, num_features, eps=1e-05, momentum=0.1, affine=True, track_running_stats=True):
        super().__init__(num_features, eps, momentum, affine, track_running_stats)
        self.scheme = QScheme("batchnorm") if config.single_precision else None

    def _native_takes(self, input):
        return (config.native_layers() and config.bn_backward_from_packed and input.is_cuda and input.dim() == 2
                and input.dtype == torch.float32 and input.size(1) % 4 == 0 and input.size(0) >= 1024
                and (self.weight is None or self.weight.dtype == torch.float32))

    def takes_activation(self, input):
        """Whether the ReLU and dropout behind this module can run in its node."""
        return self.training and self._native_takes(input) and input.size(1) <= 4096

    def forward(self, input):
        if not self.training:
            return super().forward(input)
        return self._normalise(input)

    def _normalise(self, input, dropout=None):
        """The training forward; `dropout`: the probability of the ReLU + dropout to apply as well, where takes_activation allows it."""
        self._check_input_dim(input)
        exponential_average_factor = 0.0 if self.momentum is None else self.momentum
        if self.training and self.track_running_stats and self.num_batches_tracked is not None:
            self.num_batches_tracked = self.num_batches_tracked + 1
            if self.momentum is None:
                exponential_average_factor = 1.0 / float(self.num_batches_tracked)
            else:
                exponential_average_factor = self.momentum
        bn_training = True
        if self._native_takes(input):
            # fewer rows: the framework's one-launch kernels are as fast
            track = self.track_running_stats
            args = (input, self.weight, self.bias, self.running_mean if track else None, self.running_var if track else None,
                    exponential_average_factor, self.eps, config.activation_compression_bits[0], config.seed,
                    config.take_offsets(1), config.row_offset)
            if dropout is not None:
                return _lib.native().batch_norm_act(*args, dropout, config.take_offsets(1))
            return _lib.native().batch_norm(*args)
        return qbatch_norm.apply(
            input,
            self.running_mean if not self.training or self.track_running_stats else None,
            self.running_var if not self.training or self.track_running_stats else None,
            self.weight, self.bias, bn_training, exponential_average_factor, self.eps, self.scheme)


_MODULE_CALL = torch.nn.Module.__call__
_FORWARDS = {cls: cls.forward for cls in (QBatchNorm1d, QReLUDropout)}


class QGCNConv(GCNConv):
    """layers.py:215-265.  The weight is [out_channels, in_channels] (layers.py:218), i.e. transposed
    with respect to the plain GCNConv."""

    def __init__(self, *args, **kwargs):
        super().__init__(*args, **kwargs)
        self.weight = Parameter(torch.empty(self.out_channels, self.in_channels))
        self.msg_and_aggr_func = QMatmul(self.aggr)
        self.lin_scheme = QScheme("linear") if config.single_precision else None
        self.reset_parameters()

    def forward(self, x, edge_index, edge_weight=None):
        adj_t = self._norm(edge_index)
        if self.training and config.native_layers() and self._native_takes(adj_t, x):
            # linear, aggregation and bias as one autograd node; the same compressed tensor and noise as the nodes below
            st, kept = adj_t.storage, config.kept_columns(x.size(1))
            return _lib.native().gcn(x, self.weight, self.bias, st.native_graph("sum"), config.activation_compression_bits[0],
                                     kept, config.seed, config.take_offsets(2 if kept else 1), config.row_offset,
                                     config.fused_rp, torch.is_autocast_enabled("cuda"))
        if not self.training and not torch.is_grad_enabled() and config.linear_tensor_core and self._native_takes(adj_t, x):
            return _lib.native().gcn_eval(x, self.weight, self.bias, adj_t.storage.native_graph(None),
                                          torch.is_autocast_enabled("cuda"))
        if self.training:
            # layers.py:252 passes lin_scheme in the `randmat` slot; the call is equivalent to this one.
            x = qlinear.apply(x, self.weight, None, None, None, self.lin_scheme, True)
        else:
            x = F.linear(x, self.weight, None)
        out = self.message_and_aggregate(adj_t, x)
        if self.bias is not None:
            out = out + self.bias
        return out

    def _native_takes(self, adj_t, x):
        """One GPU's graph without a gradient to its edge values, summed, with enough rows for the tensor-core kernels."""
        if not isinstance(adj_t, SparseTensor) or self.msg_and_aggr_func.reduce != "sum":
            return False
        value = adj_t.storage._value
        return (x.is_cuda and x.dim() == 2 and x.size(0) >= 1024 and self.weight.dtype == torch.float32
                and (value is None or not value.requires_grad or not torch.is_grad_enabled())
                and (x.dtype == torch.float32 or torch.is_autocast_enabled("cuda")))

    def message_and_aggregate(self, adj_t, x):
        return self.msg_and_aggr_func(adj_t, x)


class QSAGEConv(SAGEConv):
    """layers.py:123-178: the input is projected and quantised once and that one compressed copy is
    shared by the aggregation and by lin_r."""

    def __init__(self, *args, **kwargs):
        super().__init__(*args, **kwargs)
        in_channels = self.in_channels
        if isinstance(in_channels, int):
            in_channels = (in_channels, in_channels)
        bias = self.lin_l.bias is not None
        self.lin_l = QLinear(in_channels[0], self.out_channels, bias=bias, rp=True)
        if self.root_weight:
            self.lin_r = QLinear(in_channels[1], self.out_channels, bias=False, rp=True)
        self.msg_and_aggr_func = QMatmul(self.aggr)
        self.scheme = QScheme("sage") if config.single_precision else None
        self.reset_parameters()

    def forward(self, x, edge_index, size=None):
        if isinstance(x, Tensor):
            x = (x, x)
            l_eq_r = True
        else:
            l_eq_r = False
        if l_eq_r and self.training and not self.normalize and sage_layer_applies(edge_index):
            if config.native_layers() and self._native_takes(edge_index, x[0]):
                kept = config.kept_columns(x[0].size(1))
                return _lib.native().sage(x[0], self.lin_l.weight, self.lin_l.bias,
                                          self.lin_r.weight if self.root_weight else None,
                                          edge_index.storage.native_graph(self.msg_and_aggr_func.reduce),
                                          self.msg_and_aggr_func.reduce == "mean", config.activation_compression_bits[0], kept,
                                          config.seed, config.take_offsets(4 if kept else 2), config.row_offset, config.fused_rp,
                                          config.aggregate_projected_first, config.aggregate_gradient_first)
            return qsage_layer.apply(edge_index, x[0], self.lin_l.weight, self.lin_l.bias,
                                     self.lin_r.weight if self.root_weight else None,
                                     self.msg_and_aggr_func.reduce, self.scheme, self.lin_l.scheme)
        if (l_eq_r and not self.training and not self.normalize and not torch.is_grad_enabled() and config.linear_tensor_core
                and self._native_takes(edge_index, x[0])):
            return _lib.native().sage_eval(x[0], self.lin_l.weight, self.lin_l.bias, self.lin_r.weight if self.root_weight else None,
                                           edge_index.storage.native_graph(None), self.msg_and_aggr_func.reduce == "mean",
                                           torch.is_autocast_enabled("cuda"))
        if l_eq_r and self.training:
            quantized, randmat, _ = project_and_quantize(x[0], self.scheme, True)
        else:
            quantized, randmat = None, None
        out = self.message_and_aggregate(edge_index, x, quantized=quantized, randmat=randmat)
        out = self.lin_l(out)
        x_r = x[1]
        if self.root_weight and x_r is not None:
            out = out + self.lin_r(x_r, quantized, randmat)
        if self.normalize:
            out = F.normalize(out, p=2.0, dim=-1)
        return out

    def _native_takes(self, adj_t, x):
        return (isinstance(adj_t, SparseTensor) and self.msg_and_aggr_func.reduce in ("sum", "mean") and x.is_cuda
                and x.dim() == 2 and x.size(0) >= 1024 and self.lin_l.weight.dtype == torch.float32
                and (x.dtype == torch.float32 or torch.is_autocast_enabled("cuda")))

    def message_and_aggregate(self, adj_t, x, quantized=None, randmat=None):
        return self.msg_and_aggr_func(adj_t, x[0], quantized=quantized, randmat=randmat)

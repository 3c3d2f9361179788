"""Batch norm, ReLU and dropout as one node: the outputs, statistics and gradients of the separate nodes, bit for bit."""
import pytest
import torch

from exact_b200 import config
from exact_b200.layers import QBatchNorm1d, QReLUDropout, norm_act

pytestmark = pytest.mark.gpu


def run(x, g, D, p, affine, together, row_offset):
    config.compress_activation, config.row_offset = True, row_offset
    config.manual_seed(7)
    torch.manual_seed(3)
    norm, act = QBatchNorm1d(D, affine=affine).cuda().train(), QReLUDropout(p).train()
    if affine:
        torch.nn.init.uniform_(norm.weight, -0.5, 1.5)
        torch.nn.init.uniform_(norm.bias, -1, 1)
    x = x.clone().requires_grad_()
    out = norm_act(norm, act, x) if together else act(norm(x))
    offset = config.next_offset()
    out.backward(g)
    config.row_offset = 0
    assert ("Bn" in out.grad_fn.name()) == together
    return [out.detach(), x.grad, norm.running_mean, norm.running_var, torch.tensor(offset)] + [q.grad for q in norm.parameters()]


# widths whose columns come back after 1, 25, 65 and 257 runs of 256 elements; a last run that is not whole
@pytest.mark.parametrize("N,D,p,bits,affine,row_offset", [(1024, 4, 0.5, 2, True, 0), (1025, 256, 0.5, 2, True, 0), (4097, 260, 0.2, 4, True, 16),
                                                          (20011, 100, 0.0, 8, False, 0), (1500, 1028, 0.5, 1, True, 8),
                                                          (70001, 64, 0.75, 2, True, 0), (1031, 4096, 1.0, 2, True, 0)])
def test_one_node_equals_three(N, D, p, bits, affine, row_offset):
    gen = torch.Generator(device="cuda").manual_seed(N + D)
    x = torch.randn(N, D, device="cuda", generator=gen) + 0.5
    x[3] = 0.25                                      # a constant row: infinite scale of its packed form
    g = torch.randn(N, D, device="cuda", generator=gen)
    saved = config.activation_compression_bits
    config.activation_compression_bits = [bits]
    try:
        for a, b in zip(run(x, g, D, p, affine, True, row_offset), run(x, g, D, p, affine, False, row_offset)):
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num())
    finally:
        config.activation_compression_bits = saved


def test_watched_and_unsupported_modules_are_called_by_themselves():
    config.compress_activation = True
    norm, act, seen = QBatchNorm1d(64).cuda().train(), QReLUDropout(0.5).train(), []
    x = torch.randn(2048, 64, device="cuda", requires_grad=True)
    assert "Bn" in norm_act(norm, act, x).grad_fn.name()
    hook = norm.register_forward_hook(lambda m, a, out: seen.append(out))
    out = norm_act(norm, act, x)
    assert len(seen) == 1 and "Bn" not in out.grad_fn.name()
    hook.remove()
    assert "Bn" not in norm_act(norm, torch.nn.ReLU(), x).grad_fn.name()
    assert "Bn" not in norm_act(norm, act, x[:100]).grad_fn.name()      # too few rows for the kernels
    assert torch.equal(norm_act(norm.eval(), act.eval(), x), torch.relu(norm(x)))

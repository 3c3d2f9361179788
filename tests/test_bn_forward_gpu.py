"""Training batch norm on exact_bn_forward, and the fp16 copy with column sums, at the edges of their tilings."""
import numpy as np
import pytest
import torch

from exact_b200 import _lib, config
from exact_b200.layers import QBatchNorm1d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("affine,track", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("N,D", [(1024, 4), (1025, 256), (4097, 260), (20011, 100), (1500, 1028)])
def test_batch_norm_forward(N, D, affine, track):
    gen = torch.Generator(device="cuda").manual_seed(N + D)
    x = torch.randn(N, D, device="cuda", generator=gen) * 0.5 + 300.0      # a mean that would cancel in E[x^2] - E[x]^2
    x[0] = -1e3                                                            # the row that some threads' sums start from
    net = QBatchNorm1d(D, affine=affine, track_running_stats=track).cuda().train()
    if affine:
        torch.nn.init.uniform_(net.weight, 0.5, 1.5)
        torch.nn.init.uniform_(net.bias, -1, 1)
    ref = torch.nn.BatchNorm1d(D, affine=affine, track_running_stats=track).cuda().double().train()
    ref.load_state_dict(net.state_dict())
    config.compress_activation = True
    launches = _lib.LAUNCHES
    y, want = net(x.requires_grad_()), ref(x.double())
    assert _lib.LAUNCHES > launches and type(y.grad_fn).__name__ != "qbatch_normBackward"
    assert (y.double() - want).abs().max() <= 2e-6 * want.abs().max() + 300 * 2.0 ** -23 / float(x.double().std(0).min())
    if track:
        assert torch.allclose(net.running_mean.double(), ref.running_mean, rtol=1e-6)
        assert torch.allclose(net.running_var.double(), ref.running_var, rtol=1e-5)
    y.sum().backward()
    assert torch.isfinite(x.grad).all()


@pytest.mark.parametrize("N,K", [(1024, 40), (3001, 47), (20000, 256), (1500, 1)])
def test_rows_half_colsum(N, K):
    g = torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(K))
    lib, pad = _lib.load(), (K + 7) // 8 * 8
    out = torch.full((N, pad), float("nan"), dtype=torch.float16, device="cuda")
    colsum = torch.empty(K, device="cuda")
    ws = torch.empty(lib.exact_rows_scale_colsum_workspace_bytes(pad), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_rows_half_colsum", 6 * N * K, _lib.ptr(g), N, K, K, _lib.ptr(out), pad, pad, _lib.ptr(colsum),
                _lib.ptr(ws), ws.numel(), _lib.stream_ptr())
    assert torch.equal(out[:, :K], g.half()) and not out[:, K:].any()
    assert np.allclose(colsum.cpu(), g.double().sum(0).cpu(), atol=4e-6 * N ** 0.5 * float(g.abs().max()))

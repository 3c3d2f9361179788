"""Evaluation is no further from fp64 than the library's fp32 products that it replaces.

A chunk of 64 columns adds eight products of heads to a truncating accumulator: what it loses on average is given back, what is left
is below 0.3 * 8 * 2^-25 of the sum; splits (2^-24 an element) and the fp32 additions of the chunks leave 1.5e-7 in all."""
import pytest
import torch
import torch.nn.functional as F

from exact_b200 import QModule, _lib, config, gcn_norm, graphs, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [False, True])
@pytest.mark.parametrize("M,K,K2,N", [(20000, 65, 0, 64), (20000, 100, 0, 256), (1025, 128, 0, 47), (20000, 256, 256, 256), (20001, 602, 0, 41),
                                      (3000, 33, 96, 16), (20000, 640, 0, 256)])
def test_chunked_products(M, K, K2, N, sign):
    gen = torch.Generator(device="cuda").manual_seed(K)
    pad = lambda k: (k + 3) // 4 * 4
    a, a2 = (torch.randn(M, pad(k), device="cuda", generator=gen)[:, :k] if k else None for k in (K, K2))
    w, w2 = (torch.randn(N, k, device="cuda", generator=gen) if k else None for k in (K, K2))
    if sign:      # all terms of one sign: the accumulator only grows
        a, a2, w, w2 = (None if t is None else t.abs_() for t in (a, a2, w, w2))
    lib, out = _lib.load(), torch.empty(M, N, device="cuda")
    ws = torch.empty(lib.exact_linear_workspace_bytes(N, K, K2), dtype=torch.uint8, device="cuda")
    part = torch.empty(lib.exact_linear_partial_bytes(N), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), M, K, pad(K), _lib.ptr(w), K, 1, _lib.ptr(a2), K2, pad(K2), _lib.ptr(w2), K2, 1,
                N, None, None, 0, 64, _lib.ptr(part), _lib.ptr(ws), _lib.ptr(out), N, _lib.stream_ptr())
    want = a.double() @ w.double().t()
    if K2:
        want += a2.double() @ w2.double().t()
    assert (out.double() - want).norm() <= 2e-7 * want.norm()
    _lib.check_status(force=True)


@pytest.mark.parametrize("model,feats,hidden,layers", [("sage", 602, 256, 3), ("gcn", 128, 256, 3), ("gcn", 300, 64, 2), ("sage", 32, 64, 2),
                                                       ("sage", 100, 48, 2)])
def test_models(model, feats, hidden, layers):
    n = 4000
    adj = graphs.build_graph("cfg4", 0, torch.device("cuda"), nodes=n)
    if model == "gcn":
        adj = gcn_norm(adj, add_self_loops=True)
    adj.fill_cache_()
    adj.to_int32_()
    torch.manual_seed(0)
    net = QModule((models.GCN if model == "gcn" else models.SAGE)(feats, hidden, 41, layers, dropout=0.0)).cuda().eval()
    x = torch.randn(n, feats, device="cuda")
    row, col, value = adj.coo()
    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    A.index_put_((row.long(), col.long()), torch.ones(col.numel(), dtype=torch.float64, device="cuda") if value is None else value.double(),
                 accumulate=True)
    if model == "sage":
        A /= A.sum(1, keepdim=True).clamp(min=1)
    want = x.double()
    for i, conv in enumerate(net.model.convs):
        if model == "gcn":
            want = A @ (want @ conv.weight.double().t()) + conv.bias.double()
        else:
            want = (A @ want) @ conv.lin_l.weight.double().t() + conv.lin_l.bias.double() + want @ conv.lin_r.weight.double().t()
        if i + 1 < layers:
            want = F.relu(want)
    errors = []
    with torch.no_grad():
        for flag in (True, False):
            config.linear_tensor_core = flag
            try:
                errors.append(float((net(x, adj).double() - want).norm() / want.norm()))
            finally:
                config.linear_tensor_core = True
    assert errors[1] < 1e-6                   # the fp64 model is the model
    assert errors[0] <= 1.1 * errors[1], errors

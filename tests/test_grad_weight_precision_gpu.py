"""Weight gradients from packed activations are fp32-class products, whatever the width and whichever nodes ask for them.

Bound against fp64 (Frobenius): heads and tails keep 22 bits of either operand and the dropped product is below 2^-24, so a term
is off by at most 3 * 2^-23 and on average by a third of that; a range of s stages is a chain of s fp32 additions whose roundings
(2^-25 on average) add up as sqrt(s / 2).  With up to 32 stages a CTA: 2^-23 + 4 * 2^-25 < 2^-22."""
import pytest
import torch
import torch.nn.functional as F

from exact_b200 import QModule, _lib, config, gcn_norm, graphs, models
from exact_b200.cpp_extension import backward_func as B
from exact_b200.cpp_extension import quantization as Q

pytestmark = pytest.mark.gpu
BOUND = 2.0 ** -22


def _case(N, k, bits, seed, relu=True):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(N, k, device="cuda", generator=gen)
    if relu:
        x.relu_()
    pk, sb, mb = Q.quantize_pack(x, bits, seed=seed, offset=0, row_offset=0)
    return (pk, bits, sb, mb), Q.unpack_single_precision(pk, bits, sb, mb, N, k)


def _rel(a, ref):
    return float((a.double() - ref).norm() / (ref.norm() + 1e-300))


def _product(g, x):
    return sum(g[i:i + 65536].double().t() @ x[i:i + 65536].double() for i in range(0, g.size(0), 65536))


def _run(g, q0, k0, q1=None, k1=0):
    out = B.grad_weight_from_packed(g, q0, k0, q1, k1)
    _lib.check_status(force=True)
    return out


# rows around a stage of 64 and a full set of CTAs, outputs around the tile of 128, columns around 16, 112 (the most at INT8), 128
# and the passes beyond, one and two activations that share a CTA or do not
@pytest.mark.parametrize("bits", [1, 2, 4, 8])
@pytest.mark.parametrize("N,O,k0,k1", [
    (1, 4, 1, 0), (63, 128, 16, 0), (64, 132, 17, 3), (65, 256, 112, 0), (130, 40, 113, 0), (1000, 256, 128, 0), (2049, 64, 129, 0),
    (64 * 148 + 1, 256, 32, 32), (5000, 128, 64, 64), (4099, 256, 65, 64), (20011, 256, 256, 0), (3001, 252, 257, 31), (777, 100, 602, 602),
    (30000, 48, 100, 28), (70000, 256, 16, 0),
])
def test_against_fp64(N, O, k0, k1, bits):
    gen = torch.Generator(device="cuda").manual_seed(N + O)
    g = torch.randn(N, O, device="cuda", generator=gen) * torch.rand(N, 1, device="cuda", generator=gen) * 1e-5
    (q0, x0), (q1, x1) = _case(N, k0, bits, 1), _case(N, max(k1, 1), bits, 2, relu=False)
    a, b = _run(g, q0, k0, q1 if k1 else None, k1)
    assert a.shape == (O, k0) and _rel(a, _product(g, x0)) < BOUND
    if k1:
        assert b.shape == (O, k1) and _rel(b, _product(g, x1)) < BOUND


@pytest.mark.parametrize("N,O,k,bits", [(169343, 256, 256, 2), (169343, 40, 256, 2), (232965, 256, 602, 2), (169343, 256, 256, 8),
                                        (169343, 256, 256, 1), (4096, 64, 128, 2)])
def test_no_further_from_fp64_than_the_library_route(N, O, k, bits):
    """The sizes of the layers whose gradients were formed by unpacking and the library's fp32 GEMM; its error differs by a few per cent
    from seed to seed, and at one bit the kernel is 8 per cent further off (1.9e-7 against 1.8e-7)."""
    g = torch.randn(N, O, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    q, x = _case(N, k, bits, 4)
    ref = _product(g, x)
    assert _rel(_run(g, q, k)[0], ref) <= 1.25 * _rel(B.rows_reduce_mm(g, x), ref)


@pytest.mark.parametrize("model,width", [("gcn", 256), ("gcn", 100), ("sage", 256)])
def test_python_and_native_nodes_agree(model, width):
    """A debugging switch sends the layers through the Python nodes: the gradients differ by fp32 reassociation only."""
    adj = graphs.build_graph("cfg4", 0, torch.device("cuda"), nodes=6000)
    if model == "gcn":
        adj = gcn_norm(adj, add_self_loops=True)
    adj.fill_cache_()
    adj.to_int32_()
    x, y = torch.randn(6000, width, device="cuda"), torch.randint(47, (6000,), device="cuda")
    grads = []
    try:
        for flag in (False, True):
            config.check_device_status = flag
            config.compress_activation, config.kept_frac, config.activation_compression_bits = True, 1.0, [2]
            config.manual_seed(3)
            torch.manual_seed(0)
            net = QModule((models.GCN if model == "gcn" else models.SAGE)(width, width, 47, 2, dropout=0.0)).cuda().train()
            F.cross_entropy(net(x, adj), y).backward()
            grads.append({n: p.grad.clone() for n, p in net.named_parameters()})
    finally:
        config.check_device_status = False
    for n in grads[0]:
        assert _rel(grads[0][n], grads[1][n].double()) < 5e-6, n


@pytest.mark.parametrize("bits", [2, 4])
def test_pointers_off_sixteen_bytes(bits):
    N, O, k = 5001, 64, 150
    q, x = _case(N, k, bits, 5)
    shifted = torch.empty(q[0].numel() + 16, dtype=q[0].dtype, device="cuda")[3:3 + q[0].numel()].copy_(q[0])
    g = torch.empty(N * O + 1, device="cuda")[1:].view(N, O).normal_()
    assert shifted.data_ptr() % 16 and g.data_ptr() % 16 and B.grad_weight_takes(g)
    assert _rel(_run(g, (shifted, *q[1:]), k)[0], _product(g, x)) < BOUND


def test_scales_constant_rows_and_non_finite_values():
    N, O, k = 3000, 64, 96
    gen = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(N, k, device="cuda", generator=gen).relu_()
    x *= torch.exp2(torch.randint(-40, 40, (N, 1), device="cuda", generator=gen).float())   # rows far apart
    x[5], x[64:128] = 0.25, 0.0                                                             # constant rows: infinite scales
    pk, sb, mb = Q.quantize_pack(x, 2, seed=1, offset=0, row_offset=0)
    xh = Q.unpack_single_precision(pk, 2, sb, mb, N, k)
    g = torch.randn(N, O, device="cuda", generator=gen) * torch.exp2(torch.randint(-60, 0, (1, O), device="cuda", generator=gen).float())
    out, ref = _run(g, (pk, 2, sb, mb), k)[0], _product(g, xh)
    assert ((out.double() - ref).norm(dim=1) < BOUND * ref.norm(dim=1)).all()               # every output in its own scale
    g[17, 3], g[1700, 9] = float("inf"), float("nan")
    bad = ~torch.isfinite(_run(g, (pk, 2, sb, mb), k)[0])
    assert bad[3].all() and bad[9].all() and bad.sum() == 2 * k                             # confined to their outputs
    mb[77] = float("nan")
    g.nan_to_num_(0, 0, 0)
    assert not torch.isfinite(_run(g, (pk, 2, sb, mb), k)[0]).any()                         # a NaN activation row reaches everything


@pytest.mark.parametrize("O,k0,k1,bits", [(256, 256, 0, 2), (256, 32, 32, 2), (128, 100, 0, 8), (64, 602, 0, 4)])
def test_same_result_whatever_the_timing_of_the_loads(O, k0, k1, bits):
    """Cold and warm operands: no role may meet a place of a ring a round early."""
    N = 64 * 148 * 6 + 7
    g = torch.randn(N, O, device="cuda")
    (q0, _), (q1, _) = _case(N, k0, bits, 1), _case(N, max(k1, 1), bits, 2)
    flush = torch.empty(64 << 20, device="cuda")
    want = _run(g, q0, k0, q1 if k1 else None, k1)
    for i in range(20):
        if i % 2:
            flush.fill_(float(i))
        got = _run(g, q0, k0, q1 if k1 else None, k1)
        assert torch.equal(got[0], want[0]) and (not k1 or torch.equal(got[1], want[1]))

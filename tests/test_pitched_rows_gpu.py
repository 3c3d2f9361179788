"""Operands whose rows lie in a wider matrix: quantise + pack and projection + pack against the contiguous calls (same bytes),
the GEMM's addend, and the padded copies of the gradient pass."""
import pytest
import torch

from exact_b200 import _lib
from exact_b200.cpp_extension import quantization as Q

pytestmark = pytest.mark.gpu


def _wide(N, D, ldx, at=0):
    gen = torch.Generator(device="cuda").manual_seed(N + D)
    return torch.randn(N, ldx, device="cuda", generator=gen)[:, at:at + D]


@pytest.mark.parametrize("bits", [1, 2, 8])
@pytest.mark.parametrize("N,D,ldx,at", [(1003, 32, 80, 0), (2049, 75, 204, 76), (130, 301, 304, 0), (77, 602, 604, 2),
                                        (65, 128, 129, 1), (9, 1024, 1030, 4)])
def test_quantize_pack_rows(N, D, ldx, at, bits):
    x = _wide(N, D, ldx, at)
    want = Q.quantize_pack(x.contiguous(), bits, seed=7, offset=3, row_offset=8)
    got = [torch.zeros_like(t) for t in want[:3]]
    got[0].copy_(want[0]).bitwise_not_()
    _lib.invoke("exact_quantize_pack_rows", 0, _lib.ptr(x), 0, N, D, ldx, bits, 7, 3, 8, *(_lib.ptr(t) for t in got),
                _lib.stream_ptr())
    assert torch.equal(got[0][:-1], want[0][:-1])
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


# odd rows of 16-bit values: pitched to an odd and an even number, off a pair, one tile to a warp and several warps to a tile
@pytest.mark.parametrize("bits", [1, 2, 4, 8])
@pytest.mark.parametrize("N,D,ldx,at", [(1003, 47, 48, 0), (2049, 101, 105, 1), (9477, 301, 304, 0), (77, 601, 605, 2), (66, 1023, 1024, 1),
                                        (65, 100, 205, 1), (24, 1, 3, 1), (9, 5, 6, 0), (16, 7, 9, 1)])
def test_quantize_pack_rows_bf16(N, D, ldx, at, bits):
    x = torch.randn(N, ldx, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N + D)).bfloat16()[:, at:at + D]
    x[N // 2] = 1.5                                   # a constant row: its tile takes the general path
    want = Q.quantize_pack(x.contiguous(), bits, seed=7, offset=3, row_offset=8)
    got = [torch.zeros_like(t) for t in want[:3]]
    got[0].copy_(want[0]).bitwise_not_()
    _lib.invoke("exact_quantize_pack_rows", 0, _lib.ptr(x), 1, N, D, ldx, bits, 7, 3, 8, *(_lib.ptr(t) for t in got), _lib.stream_ptr())
    assert torch.equal(got[0][:-1], want[0][:-1])
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("N,D,ldx,k", [(1000, 602, 604, 76), (1537, 100, 104, 13), (300, 47, 49, 8), (4096, 128, 256, 32)])
def test_projection_of_pitched_rows(N, D, ldx, k):
    x = _wide(N, D, ldx)
    R = _lib.native().rademacher(D, k, 5, 1, x)
    want = _lib.native().rp_quantize_pack(x.contiguous(), R, 2, 5, 2, 0, True)
    got = _lib.native().rp_quantize_pack(x, R, 2, 5, 2, 0, True)
    for a, b in zip(got, want):
        n = a.numel() - (a.dtype == torch.int8)      # the allocation's last byte is nobody's
        assert torch.equal(a.flatten()[:n].float(), b.flatten()[:n].float())


@pytest.mark.parametrize("N,K,O,pad", [(1025, 64, 47, 0), (2000, 100, 128, 4), (1300, 602, 256, 1)])
def test_gemm_addend(N, K, O, pad):
    a, w, add = _wide(N, K, (K + 3) // 4 * 4), _wide(O, K, K), _wide(N, O, O + pad + 3, 1)
    lib, out = _lib.load(), torch.full((N, O), float("nan"), device="cuda")
    ws = torch.empty(lib.exact_linear_workspace_bytes(O, K, 0), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), N, K, a.stride(0), _lib.ptr(w), K, 1, None, 0, 0, None, 0, 1, O, None,
                _lib.ptr(add), add.stride(0), 0, None, _lib.ptr(ws), _lib.ptr(out), O, _lib.stream_ptr())
    want = a.double() @ w.double().t() + add.double()
    assert (out.double() - want).norm() <= 5e-6 * want.norm()


@pytest.mark.parametrize("N,K", [(1024, 47), (3000, 602), (1111, 2), (1500, 1030)])
def test_padded_copies(N, K):
    g, s = _wide(N, K, K), torch.rand(N, device="cuda")
    lib, pad = _lib.load(), (K + 3) // 4 * 4
    out, copy, colsum = torch.full((N, pad), 9.0, device="cuda"), torch.full((N, pad), 9.0, device="cuda"), torch.empty(K, device="cuda")
    ws = torch.empty(lib.exact_rows_scale_colsum_workspace_bytes(pad), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_rows_scale_copy_colsum", 0, _lib.ptr(g), N, K, K, _lib.ptr(s), _lib.ptr(out), _lib.ptr(copy), pad, pad,
                _lib.ptr(colsum), _lib.ptr(ws), ws.numel(), _lib.stream_ptr())
    assert torch.equal(copy[:, :K], g) and torch.equal(out[:, :K], g * s[:, None])
    assert not copy[:, K:].any() and not out[:, K:].any()
    assert torch.allclose(colsum.double(), g.double().sum(0), atol=4e-6 * N ** 0.5 * float(g.abs().max()))


@pytest.mark.parametrize("N,K,ldg,at,scaled", [(1024, 602, 602, 0, False), (3001, 47, 47, 0, True), (1111, 1, 1, 0, False),
                                               (1500, 90, 97, 2, True), (1030, 5, 8, 1, False)])
def test_padded_rows(N, K, ldg, at, scaled):
    g, s, pad = _wide(N, K, ldg, at), torch.rand(N, device="cuda"), (K + 3) // 4 * 4
    out = torch.full((N, pad), 9.0, device="cuda")
    _lib.invoke("exact_rows_scale_colsum", 0, _lib.ptr(g), N, K, ldg, _lib.ptr(s) if scaled else None, _lib.ptr(out), pad, pad, None,
                None, 0, _lib.stream_ptr())
    assert torch.equal(out[:, :K], g * s[:, None] if scaled else g) and not out[:, K:].any()

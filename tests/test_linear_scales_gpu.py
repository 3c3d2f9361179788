"""The chunked dense GEMM where its scales, K tiles and ways of storing can go wrong: rows of very different magnitudes, zero and
non-finite rows, contractions around a multiple of 64, results of any pitch, with and without an addend."""
import numpy as np
import pytest
import torch

from exact_b200 import _lib, check_status

pytestmark = pytest.mark.gpu


def product(a, w, bias=None, addend=None, ldc=None, a2=None, w2=None):
    (M, K), N = a.shape, w.shape[0]
    lib, K2 = _lib.load(), 0 if a2 is None else a2.shape[1]
    ldc = N if ldc is None else ldc

    def rows16(x):
        if x is None:
            return None
        out = torch.full((x.shape[0], (x.shape[1] + 3) // 4 * 4), 1e30, device="cuda")    # what lies past a row is not read
        out[:, :x.shape[1]] = x
        return out
    a, a2 = rows16(a), rows16(a2)
    out = torch.full((M, ldc), 7.0, device="cuda")
    ws = torch.empty(lib.exact_linear_workspace_bytes(N, K, K2), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), M, K, a.shape[1], _lib.ptr(w), K, 1, _lib.ptr(a2), K2,
                a2.shape[1] if K2 else 0, _lib.ptr(w2), K2, 1, N, _lib.ptr(bias), _lib.ptr(addend), addend.shape[1] if addend is not None else 0,
                64, None, _lib.ptr(ws), _lib.ptr(out), ldc, _lib.stream_ptr())
    check_status()
    assert bool((out[:, N:] == 7.0).all())
    return out[:, :N]


def bound(a, w, K):
    """A head and a tail hold 22 bits of an element or 2^-39 of the largest of 64; the dropped tail products are 2^-22; a K tile's
    twelve MMAs truncate at 2^-23 of the sum so far and the tiles' sums round: 2^-20 of sum |a||w|, and K times 2^-38 of the product
    of the rows' largest elements."""
    return 2.0 ** -20 * (a.abs() @ w.abs().t()) + 2.0 ** -38 * K * a.abs().amax(1, keepdim=True) * w.abs().amax(1)


@pytest.mark.parametrize("M,K,N,ldc", [(1024, 63, 47, None), (1025, 64, 48, None), (3000, 65, 256, None), (1153, 129, 41, 44), (257, 4, 16, None),
                                       (4097, 602, 100, 104), (128, 200, 33, None), (2000, 40, 255, 256), (130, 320, 240, None)])
@pytest.mark.parametrize("extra", ["", "bias", "addend"])
def test_magnitudes_tiles_and_stores(M, K, N, ldc, extra):
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    a = torch.randn(M, K, device="cuda", generator=gen) * torch.exp2(torch.randint(-60, 40, (M, 1), device="cuda", generator=gen).float())
    a *= torch.exp2(torch.randint(-12, 1, (M, K), device="cuda", generator=gen).float())
    w = torch.randn(N, K, device="cuda", generator=gen) * torch.exp2(torch.randint(-30, 30, (N, 1), device="cuda", generator=gen).float())
    a[5], w[3] = 0.0, 0.0
    a[7] = 1e-36                                        # scaled by the largest power of two there is
    bias = torch.randn(N, device="cuda", generator=gen) if extra == "bias" else None
    addend = torch.randn(M, (N + 3) // 4 * 4, device="cuda", generator=gen) if extra == "addend" else None
    got = product(a, w, bias, addend, ldc).double()
    ref = a.double() @ w.double().t()
    more = bias.double() if bias is not None else addend[:, :N].double() if addend is not None else torch.zeros(1, device="cuda", dtype=torch.float64)
    err = (got - ref - more).abs()
    assert bool((err <= bound(a.double(), w.double(), K) + 2.0 ** -23 * (ref + more).abs() + 1e-44).all())
    if extra == "":
        assert bool((got[5] == 0).all()) and bool((got[:, 3] == 0).all())


def test_two_operands_of_different_magnitude():
    gen = torch.Generator(device="cuda").manual_seed(2)
    a, a2 = torch.randn(2000, 70, device="cuda", generator=gen), torch.randn(2000, 130, device="cuda", generator=gen) * 1e-6
    w, w2 = torch.randn(96, 70, device="cuda", generator=gen) * 1e-6, torch.randn(96, 130, device="cuda", generator=gen)
    got = product(a, w, a2=a2, w2=w2).double()
    A, W = torch.cat([a, a2], 1).double(), torch.cat([w, w2], 1).double()
    # a row of the weight has one scale for both operands
    assert bool(((got - A @ W.t()).abs() <= bound(A, W, 200)).all())


def test_non_finite_rows_stay_where_they_are():
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn(1500, 150, device="cuda", generator=gen), torch.randn(80, 150, device="cuda", generator=gen)
    clean = product(a, w)
    a[10, 3], a[700, 149], a[1499, 64] = np.inf, -np.inf, np.nan
    got, bad = product(a, w), [10, 700, 1499]
    keep = torch.ones(1500, dtype=torch.bool, device="cuda")
    keep[bad] = False
    assert torch.equal(got[keep], clean[keep]) and not bool(got[bad].isfinite().any())

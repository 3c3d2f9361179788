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


def wide_bound(a, w, K):
    """Elements keep 22 bits each, whatever else their row holds: 2^-20 of sum |a||w|, as above."""
    return 2.0 ** -20 * (a.abs() @ w.abs().t())


# one input feature beside which the others are small, and its weights as much smaller, or zero
@pytest.mark.parametrize("scale", [1e6, 1e8, 1e15])
@pytest.mark.parametrize("M,K,K2,N", [(3000, 64, 0, 256), (1409, 100, 30, 47), (100, 33, 0, 32), (2500, 602, 0, 96)])
@pytest.mark.parametrize("zero", [False, True])
def test_dominant_feature(M, K, K2, N, scale, zero):
    gen = torch.Generator(device="cuda").manual_seed(M)
    A, W = torch.randn(M, K + K2, device="cuda", generator=gen), torch.randn(N, K + K2, device="cuda", generator=gen)
    A[:, 5] *= scale
    W[:, 5] *= 0.0 if zero else 1.0 / scale
    a, a2, w, w2 = A[:, :K].contiguous(), A[:, K:].contiguous() if K2 else None, W[:, :K].contiguous(), W[:, K:].contiguous() if K2 else None
    got, ref = product(a, w, a2=a2, w2=w2).double(), A.double() @ W.double().t()
    err = (got - ref).abs()
    assert bool((err <= wide_bound(A.double(), W.double(), K + K2)).all())
    library = (torch.nn.functional.linear(A, W).double() - ref).norm()
    assert err.norm() <= 2 * library                     # 1.2e-7 against 0.9e-7 .. 4e-7


@pytest.mark.parametrize("N", [47, 64])
def test_large_rows_and_weights_stay_finite(N):
    gen = torch.Generator(device="cuda").manual_seed(N)
    a, w = torch.randn(700, 100, device="cuda", generator=gen), torch.randn(N, 100, device="cuda", generator=gen) * 1e-3
    a[3] *= 2.0 ** 122
    a[300] *= 2.0 ** 100
    a[650] *= 2.0 ** -100
    got, ref = product(a, w).double(), a.double() @ w.double().t()
    assert bool(got.isfinite().all()) and bool(((got - ref).abs() <= wide_bound(a.double(), w.double(), 100)).all())
    w[1] *= 2.0 ** 120
    a[3] *= 2.0 ** -120
    got, ref = product(a, w).double(), a.double() @ w.double().t()
    assert bool(((got - ref).abs()[ref.abs() < 2.0 ** 127] <= wide_bound(a.double(), w.double(), 100)[ref.abs() < 2.0 ** 127]).all())
    assert not bool(got[ref.abs() > 2.0 ** 128].isfinite().any())


def in_place(a, w, bias, c):
    M, K, N = a.shape[0], a.shape[1], w.shape[0]
    ws = torch.empty(_lib.load().exact_linear_workspace_bytes(N, K, 0), dtype=torch.uint8, device="cuda")
    _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), M, K, K, _lib.ptr(w), 1, N, None, 0, 0, None, 0, 1, N, _lib.ptr(bias),
                _lib.ptr(c), c.stride(0), 64, None, _lib.ptr(ws), _lib.ptr(c), c.stride(0), _lib.stream_ptr())
    check_status()
    return c


# some of the tiles only: first, last, either half of a pair, neighbours; the others keep their bits, and each is added once
@pytest.mark.parametrize("N", [41, 96, 256])
@pytest.mark.parametrize("tiles,which", [(1, [0]), (2, [1]), (5, [0, 4]), (149, [3, 148]), (700, [0, 1, 297, 298, 591, 699])])
def test_some_tiles_are_wide(tiles, which, N):
    gen = torch.Generator(device="cuda").manual_seed(tiles + N)
    M, K = 128 * tiles - 3, 132
    a, w = torch.randn(M, K, device="cuda", generator=gen), torch.randn(K, N, device="cuda", generator=gen)   # the weight transposed
    bias, c = torch.randn(N, device="cuda", generator=gen), torch.randn(M, N, device="cuda", generator=gen)
    clean = in_place(a, w.t(), bias, c.clone())
    keep = torch.ones(M, dtype=torch.bool, device="cuda")
    for t in which:
        keep[128 * t:128 * t + 128] = False
        a[128 * t + 17, 64:96] *= 2.0 ** -40            # half of a K tile of one row
    w[64:96, :] *= 2.0 ** 10
    clean_rows = in_place(torch.where(keep[:, None], a, torch.zeros((), device="cuda")), w.t(), bias, c.clone())
    got = in_place(a, w.t(), bias, c.clone())
    assert torch.equal(got[keep], clean_rows[keep]) and not torch.equal(got, clean)
    ref = a.double() @ w.double() + bias.double() + c.double()
    assert bool(((got.double() - ref).abs() <= wide_bound(a.double(), w.t().double(), K) + 2.0 ** -22 * (ref.abs() + c.abs())).all())
    assert torch.equal(in_place(a, w.t(), bias, c.clone()), got)


def test_more_rows_than_a_launch_has_bits_for():
    gen = torch.Generator(device="cuda").manual_seed(1)
    M = 128 * 1024 * torch.cuda.get_device_properties(0).multi_processor_count + 300
    a, w = torch.randn(M, 4, device="cuda", generator=gen), torch.randn(16, 4, device="cuda", generator=gen)
    a[-40:, 1:] *= 2.0 ** -50
    a[:40, 1:] *= 2.0 ** -50
    w[:, 0] = 0.0
    got = product(a, w)
    for rows in (slice(0, 1000), slice(M - 1000, M), slice(M - 301, M - 299)):
        A, W = a[rows].double(), w.double()
        assert bool(((got[rows].double() - A @ W.t()).abs() <= wide_bound(A, W, 4)).all())


# the product starts while the preparation is still writing the workspace: nothing of what was there before is used
@pytest.mark.parametrize("M,K,N", [(1024, 63, 47), (4000, 602, 256), (70000, 128, 41)])
def test_workspace_holds_anything_before(M, K, N):
    gen = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn(M, (K + 3) // 4 * 4, device="cuda", generator=gen), torch.randn(N, K, device="cuda", generator=gen)
    w2, out = w * 2.0 ** torch.arange(N, device="cuda")[:, None].float().clamp(max=20) + 1, torch.empty(M, N, device="cuda")
    want, want2 = product(a[:, :K], w), product(a[:, :K], w2)
    size = _lib.load().exact_linear_workspace_bytes(N, K, 0)
    for i in range(60):
        ws = torch.full((size,), (0, 1, 127, 255)[i // 2 % 4], dtype=torch.uint8, device="cuda")
        for b, result in ((w, want), (w2, want2)):
            _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), M, K, a.shape[1], _lib.ptr(b), K, 1, None, 0, 0, None, 0, 1, N, None,
                        None, 0, 64, None, _lib.ptr(ws), _lib.ptr(out), N, _lib.stream_ptr())
            assert torch.equal(out, result)
    check_status()


# a layer whose two weights, and their operands the other way round, differ more and more; rows of one or both weights zero
@pytest.mark.parametrize("shift", [-30, -21, -13, 0, 13, 16, 21, 30])
@pytest.mark.parametrize("M,K,K2,N", [(1300, 100, 64, 256), (2000, 7, 130, 47)])
def test_operand_pairs_of_different_magnitudes(M, K, K2, N, shift):
    gen = torch.Generator(device="cuda").manual_seed(M)
    a, a2 = torch.randn(M, K, device="cuda", generator=gen) * 2.0 ** shift, torch.randn(M, K2, device="cuda", generator=gen)
    w, w2 = torch.randn(N, K, device="cuda", generator=gen) * 2.0 ** -shift, torch.randn(N, K2, device="cuda", generator=gen)
    w[1], w2[2] = 0.0, 0.0
    w[3], w2[3] = 0.0, 0.0
    bias = torch.randn(N, device="cuda", generator=gen)
    got = product(a, w, bias, a2=a2, w2=w2).double()
    A, W = torch.cat([a, a2], 1).double(), torch.cat([w, w2], 1).double()
    ref = A @ W.t()
    assert bool(((got - ref - bias.double()).abs() <= wide_bound(A, W, K + K2) + 2.0 ** -23 * (ref + bias).abs()).all())
    assert torch.equal(got[:, 3].float(), bias[3].expand(M))
    assert (got - ref - bias.double()).norm() <= 2e-7 * ref.norm()

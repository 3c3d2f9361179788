"""exact_linear_forward on pairs of CTAs and on single ones: odd numbers of tiles, a lone tile, more tiles than CTAs, widths with
and without a whole half for each CTA, contractions in one piece and in chunks; against fp64."""
import pytest
import torch

from exact_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [0, 64])
@pytest.mark.parametrize("M,K,K2,N", [(100, 32, 0, 32), (128, 70, 0, 256), (129, 36, 0, 64), (300, 128, 128, 224), (385, 602, 0, 16),
                                      (128 * 149, 64, 0, 96), (128 * 300 + 5, 200, 100, 256), (128 * 297 - 1, 48, 0, 47)])
def test_tiles_and_widths(M, K, K2, N, chunk):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    pad = lambda k: (k + 3) // 4 * 4
    a, a2 = (torch.randn(M, pad(k), device="cuda", generator=gen)[:, :k] if k else None for k in (K, K2))
    w, w2 = (torch.randn(N, k, device="cuda", generator=gen) if k else None for k in (K, K2))
    bias = torch.randn(N, device="cuda", generator=gen)
    lib, out = _lib.load(), torch.full((M, N), float("nan"), device="cuda")
    ws = torch.empty(lib.exact_linear_workspace_bytes(N, K, K2), dtype=torch.uint8, device="cuda")
    part = torch.empty(lib.exact_linear_partial_bytes(N), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), M, K, pad(K), _lib.ptr(w), K, 1, _lib.ptr(a2), K2, pad(K2),
                    _lib.ptr(w2), K2, 1, N, _lib.ptr(bias), None, 0, chunk, _lib.ptr(part), _lib.ptr(ws), _lib.ptr(out), N,
                    _lib.stream_ptr())
    want = a.double() @ w.double().t() + bias.double()
    if K2:
        want += a2.double() @ w2.double().t()
    assert (out.double() - want).norm() <= 5e-6 * want.norm()
    assert (out.double() - want).abs().max() <= 1e-5 * want.abs().max()
    _lib.check_status(force=True)


@pytest.mark.parametrize("N", [256, 128, 47])
def test_same_result_whatever_the_timing_of_the_loads(N):
    """Cold and warm operands: the groups of warps that take alternate K tiles must not meet a stage a round early."""
    from exact_b200.cpp_extension import backward_func as B
    a, w = torch.randn(128 * 700, 256, device="cuda"), torch.randn(N, 256, device="cuda")
    flush = torch.empty(64 << 20, device="cuda")
    want = B.linear_forward(a, w)
    for i in range(20):
        if i % 2:
            flush.fill_(float(i))
        assert torch.equal(B.linear_forward(a, w), want)

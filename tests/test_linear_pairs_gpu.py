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


# rings of two (240 columns and a single CTA), three (256) and four stages; results stored as boxes and (47, and the addend) plainly;
# more than 256 columns; the weight transposed; fp16, tf32 beside it (a range too wide for fp16) and tf32 in one chain
@pytest.mark.parametrize("chunk,wide", [(0, False), (64, False), (64, True)])
@pytest.mark.parametrize("N,addend,transposed", [(256, False, False), (256, True, True), (240, False, True), (128, False, False), (47, False, False),
                                                 (47, True, False), (300, True, False)])
def test_same_result_whatever_the_timing_of_the_loads(N, addend, transposed, chunk, wide):
    """Cold and warm operands: the groups of warps that take alternate K tiles must not meet a stage a round early."""
    from exact_b200.cpp_extension import backward_func as B
    gen = torch.Generator(device="cuda").manual_seed(N)
    a, w = torch.randn(128 * 700, 256, device="cuda", generator=gen), torch.randn(N, 256, device="cuda", generator=gen)
    if wide:
        a[128 * 100:128 * 400, 7] *= 1e8
        w[:, 7] = 0
    if transposed:
        w = w.t().contiguous().t()
    c = torch.randn(128 * 700, N, device="cuda", generator=gen) if addend else None
    flush = torch.empty(64 << 20, device="cuda")

    def product():
        return B.linear_forward(a, w, k_chunk=chunk, out=c.clone() if addend else None, accumulate=addend)
    want, ref = product(), a.double() @ w.double().t()
    if addend:
        ref += c.double()
    assert (want.double() - ref).norm() <= (2e-7 if chunk else 3e-6) * ref.norm()
    for i in range(20):
        if i % 2:
            flush.fill_(float(i))
        assert torch.equal(product(), want)
    _lib.check_status(force=True)


def test_lone_tile_of_256_columns():
    """One CTA with a ring of two stages."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, w = torch.randn(128, 512, device="cuda", generator=gen), torch.randn(256, 512, device="cuda", generator=gen)
    ws = torch.empty(_lib.load().exact_linear_workspace_bytes(256, 512, 0), dtype=torch.uint8, device="cuda")
    ref = a.double() @ w.double().t()
    for chunk in (0, 64) * 10:
        out = torch.empty(128, 256, device="cuda")
        _lib.invoke("exact_linear_forward_strided", 0, _lib.ptr(a), 128, 512, 512, _lib.ptr(w), 512, 1, None, 0, 0, None, 0, 1, 256, None, None,
                    0, chunk, None, _lib.ptr(ws), _lib.ptr(out), 256, _lib.stream_ptr())
        assert (out.double() - ref).norm() <= (2e-7 if chunk else 5e-6) * ref.norm()
    _lib.check_status(force=True)

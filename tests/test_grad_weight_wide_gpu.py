"""exact_grad_weight_from_packed beyond one producer column per thread: up to 256 columns a pass, several passes, odd
widths whose packed rows straddle the 16-byte windows, the last stage of a ragged row count."""
import pytest
import torch

from exact_b200 import config
from exact_b200.cpp_extension import backward_func as B
from exact_b200.cpp_extension import quantization as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,O,k0,k1,bits", [
    (20000, 256, 256, 0, 2), (33, 256, 256, 0, 8), (5003, 40, 256, 0, 1), (7777, 256, 129, 0, 4), (4097, 64, 255, 0, 8),
    (6001, 256, 301, 0, 2), (3000, 128, 602, 17, 2), (1025, 4, 1, 0, 2), (9001, 256, 101, 101, 4), (1, 16, 33, 7, 1),
])
def test_columns_in_passes_and_windows(N, O, k0, k1, bits):
    gen = torch.Generator(device="cuda").manual_seed(7)
    g = torch.randn(N, O, device="cuda", generator=gen)
    qs, xs = [], []
    for k in (k0, k1):
        if k:
            x = torch.randn(N, k, device="cuda", generator=gen)
            pk, sb, mb = Q.quantize_pack(x, bits, seed=k, offset=0, row_offset=0)
            qs.append((pk, bits, sb, mb))
            xs.append(Q.unpack_single_precision(pk, bits, sb, mb, N, k))
    config.check_device_status = True
    try:
        got = B.grad_weight_from_packed(g, qs[0], k0, qs[1] if k1 else None, k1)
    finally:
        config.check_device_status = False
    for a, x, k in zip(got, xs, (k0, k1)):
        ref = g.double().t() @ x.double()
        assert a.shape == (O, k) and float((a.double() - ref).norm() / ref.norm()) < 2e-3

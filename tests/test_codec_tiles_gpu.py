"""Production noise through every shape of the pack kernels' tiles (several tiles a warp, one, several warps a tile; the last
rows and the last warp partly filled) in all three input types, and unpack of odd widths, against the CPU oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from exact_b200.cpp_extension import quantization as Q
from helpers import normal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,D", [(24, 16), (1003, 30), (65, 64), (2049, 128), (250, 47), (129, 301), (77, 602), (9, 1024), (5, 1),
                                 (19, 553), (17, 1023), (11, 1026)])
def test_pack_and_unpack(N, D, dtype, bits):
    x = torch.from_numpy(normal(N, D, 71)).to(dtype)
    if N > 9:
        x[9] = 1.5               # a constant row: infinite scale
    noise = oracle.noise_b200(5, 2, N, D)
    packed, scale, mn = Q.quantize_pack(x.cuda(), bits, seed=5, offset=2)
    out = Q.unpack_single_precision(packed, bits, scale, mn, N, D).cpu()
    if dtype == torch.float16:
        op, osc, omn = oracle.quantize_activation_f16(x.numpy(), noise, bits)
        ref = oracle.unpack_f16(op, osc, omn, N, D, bits)
    else:
        op, osc, omn, _, _ = oracle.quantize_activation(x.float().numpy(), noise, bits)
        ref = oracle.dequantize_activation(op, osc, omn, N, D, bits)
    assert np.array_equal(packed.cpu().numpy().view(np.uint8)[:-1], op)
    assert np.array_equal(scale.view(torch.int16).cpu().numpy().view(np.uint16), osc.view(np.uint16))
    assert np.array_equal(mn.view(torch.int16).cpu().numpy().view(np.uint16), omn.view(np.uint16))
    assert np.array_equal(out.numpy(), ref, equal_nan=True)


@pytest.mark.parametrize("bits", [1, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,D", [(17, 256), (41, 260), (1027, 320), (8, 384), (63, 512), (25, 516)])
def test_pack_at_the_edges_of_two_warps_a_tile(N, D, dtype, bits):
    test_pack_and_unpack(N, D, dtype, bits)


# one warp a tile with three chunks of four columns (257 - 384), five in 16-bit types (513 - 640), their neighbours, in accesses of
# four elements, two and one; 9,472 rows are where enough tiles for 148 SMs begin
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,D", [(9475, 257), (9480, 300), (9465, 300), (9473, 382), (9472, 385), (9477, 516), (9479, 602), (9473, 637),
                                 (9474, 641), (9476, 33), (9478, 66)])
def test_pack_one_warp_tiles(N, D, dtype):
    test_pack_and_unpack(N, D, dtype, 4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,D,first", [(41, 47, 1), (65, 301, 1), (19, 128, 1), (19, 128, 2), (33, 602, 1), (24, 1, 1), (16, 3, 3)])
def test_pack_of_a_view_off_its_alignment(N, D, first, dtype):
    x = torch.from_numpy(normal(N, D, 72)).to(dtype)
    base = torch.full((N * D + 8,), 1e4, dtype=dtype, device="cuda")   # neighbours that would move every range
    view = base[first:first + N * D].view(N, D)
    view.copy_(x)
    for bits in (1, 2, 4, 8):
        for a, b in zip(Q.quantize_pack(view, bits, seed=5, offset=2), Q.quantize_pack(x.cuda().clone(), bits, seed=5, offset=2)):
            a, b = (t.view(torch.int8 if t.element_size() == 1 else torch.int16) for t in (a, b))
            n = a.numel() - (a.element_size() == 1)      # the stream's last byte is never written
            assert torch.equal(a[:n], b[:n])

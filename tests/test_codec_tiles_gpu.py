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

"""Entry points that encode tensor maps, as the first thing a thread does on the device."""
import threading

import pytest
import torch

from exact_b200.cpp_extension import backward_func as B
from exact_b200.cpp_extension import quantization as Q

pytestmark = pytest.mark.gpu


def test_weight_gradient_in_a_thread_that_has_no_context():
    x, g = torch.randn(1000, 128, device="cuda"), torch.randn(1000, 64, device="cuda")
    packed, scale, mn = Q.quantize_pack(x, 2, seed=1, offset=0)
    q = (packed, 2, scale, mn)
    want = B.grad_weight_from_packed(g, q, 128)
    torch.cuda.synchronize()
    got = []

    def run():
        try:
            got.append(B.grad_weight_from_packed(g, q, 128))
            torch.cuda.synchronize()
        except Exception as e:      # noqa: BLE001 (shown by the assertion below)
            got.append(e)

    thread = threading.Thread(target=run)
    thread.start()
    thread.join()
    for a, b in zip(got[0] if isinstance(got[0], tuple) else (got[0],), want if isinstance(want, tuple) else (want,)):
        assert (a is None and b is None) or torch.equal(a, b)

"""SpMM of widths that are not whole 16-byte pieces: bit for bit the columns of the same product on a padded operand, with and
without edge values and bias, on graphs with long rows and on either side of the size from which the operand is padded."""
import pytest
import torch

from exact_b200 import graphs
from exact_b200.cpp_extension import spmm as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_values", [True, False])
@pytest.mark.parametrize("reduce", ["sum", "mean"])
@pytest.mark.parametrize("nodes,edges,K", [(20000, 150000, 47), (20000, 150000, 145), (9000, 60000, 62), (9000, 60000, 255),
                                           (5000, 40000, 66), (3000, 9000, 33), (4000, 8000, 1), (80000, 500000, 145), (80000, 500000, 128)])
def test_odd_width_is_the_padded_product(nodes, edges, K, reduce, with_values):
    adj = graphs.rmat(nodes, edges, 5, "cuda")
    adj.fill_cache_()
    rowptr, col, _ = adj.csr()
    gen = torch.Generator(device="cuda").manual_seed(K)
    val = torch.rand(col.numel(), device="cuda", generator=gen) if with_values else None
    x = torch.randn(nodes, K, device="cuda", generator=gen)
    wide = torch.zeros(nodes, (K + 3) // 4 * 4, device="cuda")
    wide[:, :K] = x
    got, want = S._spmm(rowptr, col, val, x, reduce), S._spmm(rowptr, col, val, wide, reduce)
    assert got.shape == (nodes, K) and got.is_contiguous()
    assert torch.equal(got, want[:, :K])

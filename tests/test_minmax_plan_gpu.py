"""Max / min aggregation with long rows cut into pieces, and its gradients in one pass, at the edges: pieces of one edge, ties
across pieces, rows of only -inf, empty rows, widths around a warp's columns."""
import numpy as np
import pytest
import torch

import oracle
from exact_b200 import SparseTensor, config, qmatmul
from exact_b200.cpp_extension import spmm as S
from helpers import normal

pytestmark = pytest.mark.gpu
LENGTHS = [0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 96, 97, 200, 2, 0, 500]


def _graph(n, seed):
    rng = np.random.default_rng(seed)
    rowptr = np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in LENGTHS]).astype(np.int64)
    return rowptr, col, rng.standard_normal(col.size).astype(np.float32)


@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("reduce", ["max", "min"])
@pytest.mark.parametrize("K", [1, 6, 33, 128, 132])
def test_pieces_pick_the_first_winning_edge(K, reduce, idx, monkeypatch):
    monkeypatch.setattr(config, "spmm_long_row", 32)
    rowptr, col, val = _graph(600, K)
    mat = np.round(normal(600, K, 1) * 2)              # many ties
    mat[col[rowptr[5]:rowptr[6]]] = -np.inf if reduce == "max" else np.inf
    t = lambda a: torch.from_numpy(a).to(idx).cuda()
    for v in (None, val):
        out, arg = (S.spmm_max_fw if reduce == "max" else S.spmm_min_fw)(
            t(rowptr), t(col), None if v is None else torch.from_numpy(v).cuda(), torch.from_numpy(mat.astype(np.float32)).cuda())
        ro, ra = oracle.spmm_minmax(rowptr, col, v, mat.astype(np.float32), reduce)
        assert np.array_equal(out.cpu().numpy(), ro, equal_nan=True) and np.array_equal(arg.cpu().numpy(), ra)


@pytest.mark.parametrize("reduce", ["max", "min"])
@pytest.mark.parametrize("K", [5, 130])
def test_gradients_go_to_the_winning_edges(K, reduce):
    rowptr, col, val = _graph(600, 9)
    n = 600
    adj = SparseTensor(rowptr=torch.from_numpy(np.concatenate([rowptr, np.full(n - len(LENGTHS), rowptr[-1])])).cuda(),
                       col=torch.from_numpy(col).cuda(), value=torch.from_numpy(val).cuda(), sparse_sizes=(n, n))
    adj.storage.value().requires_grad_()
    config.compress_activation, config.kept_frac, config.activation_compression_bits = True, 1.0, [8]
    config.manual_seed(1)
    x = torch.from_numpy(normal(n, K, 2)).cuda().requires_grad_()
    g = torch.from_numpy(normal(n, K, 3)).cuda()
    qmatmul(adj, x, reduce).backward(g)
    _, arg = oracle.spmm_minmax(rowptr, col, val, x.detach().cpu().numpy(), reduce)
    gx, gv = np.zeros((n, K)), np.zeros(col.size)
    xh = x.detach().cpu().numpy()
    for r in range(len(LENGTHS)):
        for c in range(K):
            e = int(arg[r, c])
            if e < col.size:
                gx[col[e], c] += val[e] * float(g[r, c])
                gv[e] += xh[col[e], c] * float(g[r, c])
    assert np.allclose(x.grad.cpu().numpy(), gx, rtol=1e-5, atol=1e-5)
    # the values' gradient reads the saved operand, quantised to 8 bits
    assert np.linalg.norm(adj.storage.value().grad.cpu().numpy() - gv) < 0.02 * np.linalg.norm(gv)

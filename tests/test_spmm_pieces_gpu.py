"""The sum kernels that overlap: pieces of long rows, rows, and the sums of the pieces, against the same order of additions on the CPU."""
import numpy as np
import pytest
import torch

import oracle
from exact_b200 import config
from exact_b200.cpp_extension import spmm as S
from helpers import normal

pytestmark = pytest.mark.gpu


def graph(n, with_values):
    rng = np.random.default_rng(n)
    length = rng.integers(0, 6, n)
    for at, long in ((0, 257), (1, 256), (5, 4500), (n // 2, 512), (n - 1, 1000), (n - 2, 7681)):
        length[at] = long
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(length, out=rowptr[1:])
    col = rng.integers(0, n, rowptr[-1])
    for r in np.nonzero(length > 256)[0]:
        col[rowptr[r]:rowptr[r + 1]].sort()
    return rowptr, col, rng.standard_normal(col.size).astype(np.float32) if with_values else None


def in_pieces(rowptr, col, val, mat, reduce, threshold):
    """Rows of at most `threshold` edges in order; longer ones as pieces of that length, added in order."""
    length = np.diff(rowptr)
    count = np.maximum(-(-length // threshold), 1)
    first = np.concatenate([[0], np.cumsum(count)])
    cut = np.repeat(rowptr[:-1], count) + (np.arange(first[-1]) - np.repeat(first[:-1], count)) * threshold
    part = oracle.spmm(np.append(cut, rowptr[-1]), col, val, mat, "sum")
    out = part[first[:-1]].copy()
    for r in np.nonzero(count > 1)[0]:
        for s in range(first[r] + 1, first[r + 1]):
            out[r] += part[s]
    return out / np.maximum(length, 1).astype(np.float32)[:, None] if reduce == "mean" else out


# 75,776 rows are where the persistent kernel takes over on 148 SMs; widths of one and several column tiles, in pieces of 4, 2 and 1
@pytest.mark.parametrize("n", [3000, 75775, 75776, 80001])
@pytest.mark.parametrize("K,with_values,reduce", [(68, True, "sum"), (256, False, "mean"), (300, True, "mean"), (66, False, "sum"),
                                                  (65, True, "sum"), (48, False, "mean"), (13, True, "sum")])
def test_pieces_rows_and_sums(n, K, with_values, reduce):
    rowptr, col, val = graph(n, with_values)
    dev = [torch.from_numpy(a).cuda() if a is not None else None for a in (rowptr, col, val)]
    mats = [normal(n, K, seed) for seed in range(3)]
    outs = [S._spmm(dev[0], dev[1], dev[2], torch.from_numpy(m).cuda(), reduce) for m in mats]   # back to back
    for m, out in zip(mats, outs):
        assert np.array_equal(out.cpu().numpy(), in_pieces(rowptr, col, val, m, reduce, int(config.spmm_long_row)))

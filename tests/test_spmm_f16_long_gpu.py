"""The fp16 SpMM's long-row kernel and its column pieces at the edges of their ranges, bit for bit against the fp16
oracle: rows around one, four and more ring chunks of 64 edges, widths around 64-column blocks and 16-byte pieces."""
import numpy as np
import pytest
import torch

import oracle
from exact_b200 import config
from exact_b200.cpp_extension import spmm as S
from helpers import normal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reduce,with_values", [("sum", True), ("mean", False)])
@pytest.mark.parametrize("K", [1, 8, 23, 64, 65, 136, 264])
def test_long_rows_of_every_chunk_count(K, reduce, with_values, monkeypatch):
    monkeypatch.setattr(config, "spmm_long_row", 4)      # rows above 16 edges are chained by pairs of warps
    lengths = [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 192, 193, 255, 256, 257, 320, 321, 700, 3, 0]
    rng = np.random.default_rng(K)
    n = 800
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lengths]).astype(np.int64)
    val = rng.standard_normal(col.size).astype(np.float16) if with_values else None
    mat = normal(n, K, 3).astype(np.float16)
    ref = oracle.spmm_f16(rowptr, col, val, mat, reduce)
    out = S._spmm(torch.from_numpy(rowptr).int().cuda(), torch.from_numpy(col).int().cuda(),
                  None if val is None else torch.from_numpy(val).cuda(), torch.from_numpy(mat).cuda(), reduce)
    assert np.array_equal(out.cpu().numpy().view(np.uint16), ref.view(np.uint16))

"""Both gradients of a weighted aggregation from one walk of the transposed structure, against the oracle's separate ones."""
import numpy as np
import pytest
import torch

import oracle
from exact_b200 import SparseTensor, _lib, config, dequantize_activation, qmatmul, quantize_activation
from helpers import normal

pytestmark = pytest.mark.gpu


def hub_graph(n, seed):
    """Rows and columns of up to 300 - 900 edges (pieces), of every small length, and empty ones."""
    rng = np.random.default_rng(seed)
    r = np.concatenate([np.full(900, 7), rng.integers(0, n, 700), rng.integers(0, n // 2, 9 * n)])
    c = np.concatenate([rng.integers(0, n, 900), np.full(700, 11), rng.integers(0, n // 3, 9 * n)])
    key = np.unique(r * n + c)
    return key // n, key % n


def calls_of(run):
    """Library calls of run() by name."""
    native = _lib.native()
    native.set_timing(True)
    try:
        run()
        return [c[0] for c in native.take_calls()]
    finally:
        native.set_timing(False)


def graph_of(row, col, val, shape, idx):
    t = torch.from_numpy
    v = t(val).cuda().requires_grad_()
    adj = SparseTensor(row=t(row).cuda(), col=t(col).cuda(), value=v, sparse_sizes=shape, is_sorted=True)
    adj.fill_cache_()
    return v, adj.to_int32_() if idx == torch.int32 else adj


def check_both_gradients(row, col, shape, K, reduce, idx, g):
    """Against the oracle's gradients from the operand as it is saved (8 bits); g: numpy, or a torch tensor on the GPU."""
    n_rows, n_cols = shape
    rowptr, colptr = np.zeros(n_rows + 1, np.int64), np.zeros(n_cols + 1, np.int64)
    np.cumsum(np.bincount(row, minlength=n_rows), out=rowptr[1:])
    np.cumsum(np.bincount(col, minlength=n_cols), out=colptr[1:])
    val = np.random.default_rng(1).standard_normal(col.size).astype(np.float32)
    v, adj = graph_of(row, col, val, shape, idx)
    x = torch.from_numpy(normal(n_cols, K, 6)).cuda().requires_grad_()
    config.compress_activation, config.kept_frac = True, 1.0
    saved, config.activation_compression_bits = config.activation_compression_bits, [8]
    try:
        config.manual_seed(4)
        q = quantize_activation(x.detach(), None)
        mat = dequantize_activation(q, tuple(x.shape)).cpu().numpy()
        config.manual_seed(4)
        names = calls_of(lambda: qmatmul(adj, x, reduce).backward(g if isinstance(g, torch.Tensor) else torch.from_numpy(g).cuda()))
    finally:
        config.activation_compression_bits = saved
    assert ("exact_spmm_weighted_backward" in names) == (K <= 256) and ("exact_spmm_value_bw" in names) == (K > 256)
    g = g.cpu().numpy() if isinstance(g, torch.Tensor) else g
    assert np.array_equal(v.grad.cpu().numpy(), oracle.spmm_value_bw(rowptr, col, mat, g, reduce), equal_nan=True)
    perm = np.argsort(col * n_rows + row, kind="stable")
    w = val[perm]
    if reduce == "mean":
        w = w / np.maximum(np.diff(rowptr), 1)[row[perm]].astype(np.float32)
    ref = oracle.spmm(colptr, row[perm], w, g, "sum")
    got, long = x.grad.cpu().numpy(), np.diff(colptr) > int(config.spmm_long_row)
    assert np.array_equal(got[~long], ref[~long], equal_nan=True)
    # long rows are summed in pieces of 256 edges: two orders of n fp32 multiply-adds, each within n * 2^-24 of the sum of magnitudes
    size = oracle.spmm(colptr, row[perm], np.abs(w), np.abs(np.nan_to_num(g, posinf=0)), "sum")[long]
    ok = np.isfinite(ref[long])
    assert (np.abs(got[long] - ref[long])[ok] <= (2 * np.diff(colptr)[long, None] * 2.0 ** -24 * size)[ok]).all()
    return long.any()


# columns: every number of 32-column groups with and without a remainder, and one width beyond the kernel's range
@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("K", [1, 31, 32, 33, 64, 100, 128, 160, 192, 200, 224, 250, 256, 260])
@pytest.mark.parametrize("reduce", ["sum", "mean"])
def test_both_gradients_in_one_walk(K, reduce, idx):
    n = 2000
    row, col = hub_graph(n, K)
    g = normal(n, K, 7)
    if K > 1:
        g[5, K - 1] = np.inf                   # stays in its row's edges and its column
    assert check_both_gradients(row, col, (n, n), K, reduce, idx, g)


# adjacencies that are not square, with empty rows and columns, and gradients that are transposed, sliced or expanded
@pytest.mark.parametrize("shape", [(2000, 700), (700, 2000), (2000, 2000)])
@pytest.mark.parametrize("K,layout", [(40, "transposed"), (97, "sliced"), (128, "expanded"), (5, "transposed")])
@pytest.mark.parametrize("reduce", ["sum", "mean"])
def test_rectangular_and_strided(shape, K, layout, reduce):
    row, col = hub_graph(2000, K)
    keep = (row < shape[0]) & (col < shape[1])
    row, col = row[keep], col[keep]
    base = torch.from_numpy(normal(shape[0], K, 7)).cuda()
    if layout == "transposed":
        g = base.t().contiguous().t()
    elif layout == "sliced":
        g = torch.cat([base, base], 1)[:, 3:3 + K]
    else:
        g = base[0].expand(shape[0], K)
    assert not g.is_contiguous()
    check_both_gradients(row, col, shape, K, reduce, torch.int64, g)


# nothing saved compressed: the Python nodes and their separate kernels
@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("K", [1, 31, 32, 33, 64, 100, 128, 160, 192, 200, 224, 250, 256, 260])
@pytest.mark.parametrize("reduce", ["sum", "mean"])
def test_both_gradients(K, reduce, idx):
    n = 2000
    row, col = hub_graph(n, K)
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(row, minlength=n), out=rowptr[1:])
    val = np.random.default_rng(1).standard_normal(col.size).astype(np.float32)
    t = torch.from_numpy
    v = t(val).cuda().requires_grad_()
    adj = SparseTensor(row=t(row).cuda(), col=t(col).cuda(), value=v, sparse_sizes=(n, n), is_sorted=True)
    adj.fill_cache_()
    if idx == torch.int32:
        adj.to_int32_()
    mat, g = normal(n, K, 6), normal(n, K, 7)
    if K > 1:
        g[5, K - 1] = np.inf                   # stays in its row's edges and its column
    x = t(mat).cuda().requires_grad_()
    config.compress_activation = False
    try:
        qmatmul(adj, x, reduce).backward(t(g).cuda())
    finally:
        config.compress_activation = True
    assert np.array_equal(v.grad.cpu().numpy(), oracle.spmm_value_bw(rowptr, col, mat, g, reduce), equal_nan=True)
    perm = np.argsort(col * n + row, kind="stable")
    w = val[perm]
    if reduce == "mean":
        w = w / np.maximum(np.diff(rowptr), 1)[row[perm]].astype(np.float32)
    colptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(col, minlength=n), out=colptr[1:])
    ref = oracle.spmm(colptr, row[perm], w, g, "sum")
    got, long = x.grad.cpu().numpy(), np.diff(colptr) > int(config.spmm_long_row)
    assert long.any() and np.array_equal(got[~long], ref[~long], equal_nan=True)
    ok = np.isfinite(ref[long])
    # pieces of 256 edges: a regrouped sum of fp32 terms, 1e-5 of the row's largest entry as elsewhere
    assert np.abs((got[long] - ref[long])[ok]).max() <= 1e-5 * np.abs(ref[long][ok]).max()


def test_one_gradient_at_a_time_takes_the_separate_kernels():
    n, K = 2000, 64
    row, col = (torch.from_numpy(a).cuda() for a in hub_graph(n, 3))
    val = torch.rand(col.numel(), device="cuda")
    mat, g = (torch.from_numpy(normal(n, K, s)).cuda() for s in (6, 7))

    def grads(x_rg, v_rg):
        v, x = val.clone().requires_grad_(v_rg), mat.clone().requires_grad_(x_rg)
        adj = SparseTensor(row=row, col=col, value=v, sparse_sizes=(n, n), is_sorted=True)
        config.compress_activation = True
        config.manual_seed(1)
        qmatmul(adj, x, "sum").backward(g)
        return x.grad, v.grad

    both, only_x, only_v = grads(True, True), grads(True, False), grads(False, True)
    assert torch.equal(both[0], only_x[0]) and torch.equal(both[1], only_v[1])


@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
def test_no_columns_give_zero_gradients_of_the_values(idx):
    rowptr = torch.tensor([0, 2, 2, 5], dtype=idx, device="cuda")
    col, perm = torch.tensor([0, 1, 1, 2, 3], dtype=idx, device="cuda"), torch.tensor([3, 0, 1, 4, 2], dtype=idx, device="cuda")
    val, out = torch.ones(5, device="cuda"), torch.full((6,), 7.0, device="cuda")
    p = _lib.ptr
    _lib.invoke("exact_spmm_weighted_backward", 0, p(rowptr), p(col), p(val), p(perm), None, rowptr.element_size(), None, None, 3, 0, 0,
                None, None, None, None, 0, None, None, 0, None, None, None, p(out), _lib.stream_ptr())
    assert out.tolist() == [0, 0, 0, 0, 0, 7]
    n = 500
    poison = torch.full((3 * n,), float("nan"), device="cuda")   # what the allocator hands out next
    v = torch.rand(3 * n, device="cuda").requires_grad_()
    row = torch.arange(3 * n, device="cuda") // 3
    adj = SparseTensor(row=row, col=(row * 7 + torch.arange(3 * n, device="cuda")) % n, value=v, sparse_sizes=(n, n))
    x = torch.empty(n, 0, device="cuda").requires_grad_()
    y = qmatmul(adj, x, "sum")
    del poison
    y.backward(torch.empty_like(y))
    assert not bool(v.grad.any()) and x.grad.shape == x.shape


def short_rows(n, per_row, hubs, seed):
    """n rows of per_row edges each way (a few less: duplicates), and `hubs` columns of 300 edges."""
    rng = np.random.default_rng(seed)
    r = np.concatenate([np.tile(np.arange(n), per_row), rng.integers(0, n, 300 * hubs)])
    c = np.concatenate([np.concatenate([rng.permutation(n) for _ in range(per_row)]), np.repeat(rng.integers(0, n, hubs), 300)])
    key = np.unique(r * n + c)
    return key // n, key % n


# either side of every line of the rule, and the same bits on both
@pytest.mark.parametrize("n,per_row,hubs,K,joint", [(65536, 3, 0, 16, False), (65535, 3, 0, 16, True), (70000, 3, 0, 64, True), (70000, 9, 0, 16, True),
                                                    (70000, 3, 0, 3, True), (70000, 3, 30, 16, True), (70000, 3, 8, 16, False),
                                                    (1 << 20, 2, 0, 3, False), (1 << 18, 3, 40, 8, False), (1 << 18, 6, 40, 8, True)])
def test_short_narrow_rows_keep_the_separate_kernels(n, per_row, hubs, K, joint):
    row, col = short_rows(n, per_row, hubs, K)
    val = np.random.default_rng(1).random(col.size, dtype=np.float32)
    g, mat = torch.from_numpy(normal(n, K, 7)).cuda(), torch.from_numpy(normal(n, K, 6)).cuda()
    config.compress_activation = True
    grads = []
    for x_rg, v_rg in ((True, True), (True, False), (False, True)):
        v, adj = graph_of(row, col, val, (n, n), torch.int64)
        v.requires_grad_(v_rg)
        x = mat.clone().requires_grad_(x_rg)
        config.manual_seed(2)
        names = calls_of(lambda: qmatmul(adj, x, "sum").backward(g))
        assert ("exact_spmm_weighted_backward" in names) == (joint and x_rg and v_rg)
        grads.append((x.grad, v.grad))
    assert torch.equal(grads[0][0], grads[1][0]) and torch.equal(grads[0][1], grads[2][1])

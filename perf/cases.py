"""What this framework's users have it compute, as cases that can be timed and compared.

Three kinds of work, all through the public entry points of `exact_b200`:

  compress / decompress   quantize_activation / dequantize_activation on one saved activation
  aggregate               qmatmul (the adjacency times a dense operand), forward and backward
  train / infer           a QModule-converted GCN or GraphSAGE on a whole graph: one training step up to the
                          parameter gradients, or one evaluation pass

Sizes are the repository's benchmark configurations (exact_b200.graphs.CONFIGS) and the grid of its kernel sweep."""
import math

import torch
import torch.nn.functional as F

import exact_b200 as E
from exact_b200 import graphs, models

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
SIZE = {"fp32": 4, "bf16": 2, "fp16": 2}
LOSS_SCALE = 65536.0   # what torch.amp.GradScaler starts with


def _codec(kind, name, rows, cols, bits, dtype):
    return {"name": name, "kind": kind, "rows": rows, "cols": cols, "bits": bits, "dtype": dtype}


def _model(kind, name, cfg, **other):
    """A case of a benchmark configuration: `edges` counts sampled undirected edges."""
    c = graphs.CONFIGS[cfg]
    edges = c["undirected"] if "undirected" in c else int(c["nodes"] * c["avg_degree"] / 2)
    case = {"name": name, "kind": kind, "model": c["model"], "graph": c["graph"], "nodes": c["nodes"], "edges": edges,
            "self_loops": c["self_loops"], "index": "int32", "feats": c["feats"], "hidden": c["hidden"],
            "classes": c["classes"], "layers": c["layers"], "batch_norm": c["batch_norm"], "dropout": c["dropout"],
            "bits": c["bits"], "kept_frac": c["kept_frac"], "amp": False}
    case.update(other)
    return case


def _aggregate(name, graph, nodes, edges, index, cols, reduce, weighted, bits):
    return {"name": name, "kind": "aggregate", "graph": graph, "nodes": nodes, "edges": edges, "self_loops": True,
            "index": index, "cols": cols, "reduce": reduce, "weighted": weighted, "bits": bits, "kept_frac": 1.0}


def listed():
    return [
        # One activation of a small graph: the call's latency is what the user sees.
        _codec("compress", "compress_small", 4096, 128, 2, "fp32"),
        # The shape the pack / unpack bandwidths are quoted on.
        _codec("compress", "compress_1m", 1_000_000, 128, 2, "fp32"),
        _codec("decompress", "decompress_1m", 1_000_000, 128, 2, "fp32"),
        # Input features of the reddit-shaped configuration held in bf16: 602 columns, an odd number of rows.
        _codec("compress", "compress_reddit_bf16", 232_965, 602, 4, "bf16"),
        # A hidden activation of the arxiv-shaped configuration saved at 8 bits.
        _codec("decompress", "decompress_hidden_int8", 169_343, 256, 8, "fp32"),
        # Learned edge weights: forward, the operand's gradient and the weights' gradient.
        _aggregate("aggregate_weighted", "rmat", 169_343, 1_166_243, "int64", 128, "sum", True, 2),
        # The smallest training step (int64 indices, as a loader delivers them): launches and host time count.
        _model("train", "train_gcn_4k", "cfg1", index="int64"),
        # The arxiv-shaped GCN with batch norm, in fp32 and under autocast with a scaled loss.
        _model("train", "train_gcn_arxiv", "cfg2"),
        _model("train", "train_gcn_arxiv_amp", "cfg2", amp=True),
        # The GraphSAGE configurations with random projection: wide input features, and the largest graph.
        _model("train", "train_sage_reddit", "cfg3"),
        _model("train", "train_sage_products", "cfg4"),
        # The evaluation pass that a training program runs every few epochs.
        _model("infer", "infer_sage_reddit", "cfg3"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["compress", "decompress", "aggregate", "train", "train", "infer"])
    if kind in ("compress", "decompress"):
        cols = _log(rng, 16, 1024)
        rows = _log(rng, 1000, min(3_000_000, 600_000_000 // cols))
        if rng.random() < 0.5:
            cols = max(16, cols // 16 * 16)   # layer widths; the others are feature counts as data sets have them
        case = _codec(kind, "", rows, cols, rng.choice([1, 2, 2, 4, 8]), rng.choice(["fp32", "fp32", "bf16", "fp16"]))
        del case["name"]
        return case
    nodes = _log(rng, 2000, 500_000)
    edges = min(15_000_000, int(nodes * math.exp(rng.uniform(math.log(3), math.log(60)))))
    if kind == "aggregate":
        weighted = rng.random() < 0.4
        case = _aggregate("", "rmat", nodes, edges, rng.choice(["int32", "int64"]), _log(rng, 16, 256),
                          rng.choice(["sum", "mean", "max", "min"]), weighted, rng.choice([2, 4, 8]))
        del case["name"]
        return case
    model = rng.choice(["gcn", "sage"])
    case = _model(kind, "", "cfg2" if model == "gcn" else "cfg4", nodes=nodes, edges=edges,
                  graph=rng.choice(["rmat", "rmat", "er"]), self_loops=model == "gcn" or rng.random() < 0.5,
                  index=rng.choice(["int32", "int64"]), feats=_log(rng, 32, 640), hidden=rng.choice([64, 128, 256]),
                  classes=_log(rng, 7, 112), layers=rng.choice([2, 3]), batch_norm=rng.random() < 0.5,
                  dropout=rng.choice([0.0, 0.2, 0.5]), bits=rng.choice([1, 2, 2, 4, 8]),
                  kept_frac=rng.choice([1.0, 0.5, 0.125]), amp=rng.random() < 0.25)
    del case["name"]
    return case


def _configure(case, seed):
    E.config.compress_activation = True
    E.config.activation_compression_bits = [case["bits"]]
    E.config.kept_frac = case.get("kept_frac", 1.0)
    E.config.row_offset = 0
    E.config.manual_seed(seed)


def _graph(case, seed):
    if case["graph"] == "er":
        return graphs.erdos_renyi(case["nodes"], 2 * case["edges"] / case["nodes"], seed, "cuda", case["self_loops"])
    return graphs.rmat(case["nodes"], case["edges"], seed, "cuda", self_loops=case["self_loops"])


def _nnz(case):
    nnz = 2 * case["edges"] + (case["nodes"] if case["self_loops"] else 0)
    return int(0.88 * nnz) if case.get("weighted") else nnz


def _thinned(adj, nnz, gen):
    """`nnz` of the edges: the generator's own count depends on the seed, and a weights' gradient has its length."""
    row, col, _ = adj.coo()
    keep = torch.randperm(col.numel(), device="cuda", generator=gen)[:nnz].sort()[0]
    assert keep.numel() == nnz
    return E.SparseTensor(row=row[keep], col=col[keep], sparse_sizes=adj.sparse_sizes(), is_sorted=True)


def _ready(adj, case, reduce):
    """The index structures a training program builds once and keeps with its graph."""
    adj.fill_cache_()
    if case["index"] == "int32":
        adj.to_int32_()
    if reduce in ("sum", "mean"):
        adj.storage.transposed(reduce)
    return adj


def prepare(case, seed):
    _configure(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    kind = case["kind"]
    if kind in ("compress", "decompress"):
        # what a ReLU leaves of a normal activation
        x = torch.randn(case["rows"], case["cols"], device="cuda", generator=gen).relu_().to(DTYPES[case["dtype"]])
        if kind == "compress":
            return {"kind": kind, "seed": seed, "x": x}
        return {"kind": kind, "shape": x.shape, "quantized": E.quantize_activation(x, None)}
    adj = _graph(case, seed)
    n = adj.size(0)
    if kind == "aggregate":
        if case["weighted"]:
            adj = _thinned(adj, _nnz(case), gen)
            adj = adj.set_value(torch.rand(adj.nnz(), device="cuda", generator=gen).add_(0.1))
        _ready(adj, case, None if case["weighted"] else case["reduce"])
        if case["weighted"]:
            adj.storage.value().requires_grad_()
        x = torch.randn(n, case["cols"], device="cuda", generator=gen).requires_grad_()
        return {"kind": kind, "seed": seed, "adj": adj, "x": x, "reduce": case["reduce"],
                "grad": torch.randn(n, case["cols"], device="cuda", generator=gen)}
    if case["model"] == "gcn":
        adj = E.gcn_norm(adj, add_self_loops=False)
    _ready(adj, case, "sum" if case["model"] == "gcn" else "mean")
    cls = models.GCN if case["model"] == "gcn" else models.SAGE
    net = E.QModule(cls(case["feats"], case["hidden"], case["classes"], case["layers"], dropout=case["dropout"],
                        batch_norm=case["batch_norm"])).cuda().train(kind == "train")
    # A convolution's bias in front of a batch norm has gradient zero: what is computed for it is rounding.
    no_grad = ["convs.%d.%s" % (i, b) for i in range(case["layers"] - 1) for b in ("bias", "lin_l.bias")]
    params = {k: p for k, p in net.model.named_parameters() if not (case["batch_norm"] and k in no_grad)}
    return {"kind": kind, "seed": seed, "adj": adj, "net": net, "params": params, "amp": case["amp"],
            "x": torch.randn(n, case["feats"], device="cuda", generator=gen),
            "y": torch.randint(case["classes"], (n,), device="cuda", generator=gen)}


def run(state):
    kind = state["kind"]
    if kind == "decompress":
        return E.dequantize_activation(state["quantized"], state["shape"])
    E.config.manual_seed(state["seed"])   # a reproducible run: the noise is keyed by the seed and the call order
    if kind == "compress":
        packed, _, scale, mn = E.quantize_activation(state["x"], None)
        return packed[:-1], scale, mn     # the stream's last byte is allocated and never written
    adj, x = state["adj"], state["x"]
    if kind == "aggregate":
        x.grad = None
        value = adj.storage.value()
        if value is not None:
            value.grad = None
        out = E.qmatmul(adj, x, state["reduce"])
        out.backward(state["grad"])
        return out, x.grad, None if value is None else value.grad
    net = state["net"]
    if kind == "infer":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.float16, enabled=state["amp"]):
            return net(x, adj)
    net.zero_grad(set_to_none=True)
    with torch.autocast("cuda", dtype=torch.float16, enabled=state["amp"]):
        out = net(x, adj)
        # per-row losses and a parallel sum: nll_loss adds up its mean in one block
        loss = F.cross_entropy(out.float(), state["y"], reduction="none").sum() / out.size(0)
    (loss * LOSS_SCALE if state["amp"] else loss).backward()
    return {"loss": loss, "out": out, "grad": {k: p.grad for k, p in state["params"].items()}}


def _packed(rows, cols, bits):
    return -(-rows * bits // 8) * cols


def work(case):
    kind = case["kind"]
    if kind in ("compress", "decompress"):
        rows, cols = case["rows"], case["cols"]
        size = SIZE[case["dtype"]]
        if kind == "decompress" and case["dtype"] == "bf16":
            size = 4      # dequantised to fp32, as the statistics of bf16 and fp32 activations are the same
        return {"bytes": rows * cols * size + _packed(rows, cols, case["bits"]) + 4 * rows,
                "flops": (4 if kind == "compress" else 2) * rows * cols}
    n = case["nodes"]
    nnz = _nnz(case)
    index = 4 if case["index"] == "int32" else 8
    if kind == "aggregate":
        dense = n * case["cols"] * 4
        structure = (nnz + n + 1) * index + (nnz * 4 if case["weighted"] else 0)
        total = 2 * (2 * dense + structure)
        flops = 4 * nnz * case["cols"]
        saved = case["weighted"] or case["reduce"] in ("max", "min")   # the operand, compressed
        if saved:
            total += 2 * (_packed(n, case["cols"], case["bits"]) + 4 * n)
        if case["weighted"]:
            total += nnz * (4 + index)
            flops += 2 * nnz * case["cols"]
        return {"bytes": total, "flops": flops}
    size = 2 if case["amp"] else 4
    weighted = nnz * 4 if case["model"] == "gcn" else 0
    dense = 2 if case["model"] == "sage" else 1        # products with a weight: lin_l and lin_r, or one
    total = flops = 0
    for i in range(case["layers"]):
        a = case["feats"] if i == 0 else case["hidden"]
        b = case["classes"] if i == case["layers"] - 1 else case["hidden"]
        width = min(a, b)
        structure = (nnz + n + 1) * index + weighted
        # the aggregation needs whole columns of its operand before the first row comes out, so each layer reads
        # its input and writes its output
        total += n * (a + b) * size + structure
        flops += dense * 2 * n * a * b + 2 * nnz * width
        if kind == "train":
            kept = a if case["kept_frac"] >= 1 else int(case["kept_frac"] * a + 0.999)
            total += 2 * dense * (_packed(n, kept, case["bits"]) + 4 * n)      # saved activations, out and back
            total += n * b * size                                             # the output's gradient
            flops += dense * 2 * n * kept * b                                 # the weights' gradients
            if i > 0:
                total += n * a * size
                flops += dense * 2 * n * a * b
            if i > 0 or case["model"] == "gcn":
                total += structure
                flops += 2 * nnz * width
    return {"bytes": total, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("compress", "decompress"):
        return "exact"                       # codes and statistics are defined to the bit, given the seed
    if case.get("amp"):
        return {"rel": 1e-2, "max": 0.5}     # fp16 operands, sums rounded to fp16
    if kind in ("aggregate", "infer"):
        return {"rel": 1e-5}
    if case["kept_frac"] < 1.0:
        # the projection is a tf32 product: a few codes in a thousand of the saved activations, on which the weight
        # gradients are formed, fall on the other side of a rounding boundary
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 2e-3, "max": 0.1}         # fp32, weight gradients with tf32 operands

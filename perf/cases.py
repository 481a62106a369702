"""Performance cases of the framework: what its users run, through the entry points they call.

A case is a dict of plain values; its ``kind`` says which entry point it goes through:

  agg       one GCN / GraphSAGE aggregation on a resident block format: the ``SpMM_sr_bcrs`` drop-in
            (fp16, tf32) or ``ops.spmm`` (bf16, and e4m3 features with per-row scales)
  convert   CSR -> block format on the GPU, GCN form with values (``Block_sr_bcrs``) or GAT form with
            slot maps (``ATT_Block_v3``)
  gcn       a GCN layer, forward and backward (``layers.GCNConv``)
  attention dot-product GAT aggregation of an inference pass, fused (``gat.GATGraph.attention``)
  gat       an additive multi-head GAT layer, forward and backward, fused kernels (``gat.GATConv``)
  chain     the same layer as the reference composes it from separate ops (``layers.GATConv_multi``)
  serve     one aggregation tick of the serving loop: many graphs in one launch (``serving.BatchedSpmm``)

Graphs are power-law (Chung-Lu) graphs made on the GPU from the seed alone, symmetric and with
self-loops, as the loaders of the models make them.
"""
import math

import torch

from att_gb300 import gat, layers, ops, serving
from att_gb300.compat import ATT_Block_v3, Block_sr_bcrs, SpMM_sr_bcrs

HEADS_SLOPE = 0.2


def listed():
    return [
        # the smallest aggregation of the benchmark, 16,384 nodes: latency and launches
        {"name": "agg_small_fp16", "kind": "agg", "dtype": "fp16", "n": 16384, "deg": 10.0, "f": 64},
        # full-graph GCN aggregation at the largest node count of the benchmark
        {"name": "agg_large_fp16", "kind": "agg", "dtype": "fp16", "n": 2449029, "deg": 25.0, "f": 128},
        # the same graph with e4m3 features, the low-precision inference form
        {"name": "agg_large_fp8", "kind": "agg", "dtype": "fp8", "n": 2449029, "deg": 25.0, "f": 128},
        # fp32-accurate aggregation of a mid-size citation-like graph, 100 raw input features
        {"name": "agg_mid_tf32", "kind": "agg", "dtype": "tf32", "n": 169343, "deg": 14.0, "f": 100},
        # preprocessing: the large graph converted once per load
        {"name": "convert_large", "kind": "convert", "form": "gcn", "n": 2449029, "deg": 25.0},
        # preprocessing of a GAT training graph (slot -> edge maps, both directions)
        {"name": "convert_gat_mid", "kind": "convert", "form": "gat", "n": 169343, "deg": 14.0},
        # one GCN training layer, 100 -> 64 features
        {"name": "gcn_layer_mid", "kind": "gcn", "n": 169343, "deg": 14.0, "fin": 100, "f": 64},
        # attention over a dense social graph, about 114M edges, one head of 64
        {"name": "attention_large_fp16", "kind": "attention", "dtype": "fp16", "n": 232965, "deg": 490.0, "f": 64},
        # fp32 attention (3xTF32) on a smaller graph
        {"name": "attention_mid_fp32", "kind": "attention", "dtype": "fp32", "n": 100000, "deg": 100.0, "f": 64},
        # a hidden GAT layer of the training step, 128 -> 4 heads of 64, bf16
        {"name": "gat_layer_bf16", "kind": "gat", "dtype": "bf16", "n": 169343, "deg": 14.0, "fin": 128, "heads": 4,
         "f": 64},
        # the same layer as a chain of the separate drop-in ops, fp16
        {"name": "chain_layer_fp16", "kind": "chain", "n": 169343, "deg": 14.0, "fin": 128, "heads": 4, "f": 64},
        # a tick of the serving loop: 16 graphs of uneven sizes, 128 features
        {"name": "serve_tick", "kind": "serve", "graphs": 16, "nmax": 100000, "f": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["agg", "agg", "agg", "convert", "gcn", "attention", "attention", "gat", "chain", "serve"])
    if kind in ("agg", "convert"):
        n = _log_int(rng, 1000, 2449029)
        case = {"kind": kind, "n": n, "deg": round(rng.uniform(5.0, 25.0 if n > 1000000 else 50.0), 2)}
        if kind == "agg":
            case["dtype"] = rng.choice(["fp16", "bf16", "fp8", "tf32"])
            # whole rows of the kernels' granule for the entry points that ask for it; any width elsewhere
            case["f"] = {"fp16": lambda: rng.randint(16, 128), "bf16": lambda: 8 * rng.randint(2, 16),
                         "fp8": lambda: 16 * rng.randint(2, 8), "tf32": lambda: rng.randint(16, 128)}[case["dtype"]]()
        else:
            case["form"] = rng.choice(["gcn", "gat"])
        return case
    if kind == "gcn":
        return {"kind": kind, "n": _log_int(rng, 1000, 500000), "deg": round(rng.uniform(5.0, 50.0), 2),
                "fin": rng.randint(16, 128), "f": rng.choice([16, 32, 40, 47, 64, 128])}
    if kind == "attention":
        n = _log_int(rng, 1000, 232965)
        return {"kind": kind, "dtype": rng.choice(["fp16", "bf16", "fp32"]), "n": n,
                "deg": round(math.exp(rng.uniform(math.log(5.0), math.log(min(200.0, n / 10)))), 2),
                "f": rng.choice([32, 64, 64, 128])}
    if kind in ("gat", "chain"):
        case = {"kind": kind, "n": _log_int(rng, 1000, 200000), "deg": round(rng.uniform(5.0, 30.0), 2),
                "fin": rng.randint(8, 32) * 8, "heads": rng.choice([1, 2, 4]), "f": rng.choice([32, 64])}
        if kind == "gat":
            case["dtype"] = rng.choice(["bf16", "fp16"])
        return case
    return {"kind": kind, "graphs": rng.randint(1, 32), "nmax": _log_int(rng, 5000, 200000), "f": rng.choice([64, 128])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _graph(n, deg, seed, gamma=2.1):
    """(rows, cols) int64 on the GPU, sorted by row and column: about n * deg
    directed edges of a symmetric power-law graph and a self-loop per node; no
    node is expected to have more than n / 4 neighbours."""
    g = _gen(seed)
    pairs = max(1, int(n * deg / 2))
    w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) ** (-1.0 / (gamma - 1.0))
    w = torch.minimum(w, w.sum() * (n / (8.0 * pairs)))
    cdf = torch.cumsum((w * (2.0 ** 40 / w[0])).long(), 0)  # whole numbers: the same sums in every run
    perm = torch.randperm(n, generator=g, device="cuda")

    def ends(m):
        u = (torch.rand(m, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]).long()
        return perm[torch.searchsorted(cdf, u).clamp_(max=n - 1)]

    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    for _ in range(8):
        m = pairs - keys.numel()
        if m <= pairs // 64:
            break
        u, v = ends(m + m // 8), ends(m + m // 8)
        lo, hi = torch.minimum(u, v), torch.maximum(u, v)
        keys = torch.unique(torch.cat([keys, (lo * n + hi)[lo != hi]]))
    a, b = keys // n, keys % n
    loop = torch.arange(n, device="cuda")
    key = torch.sort(torch.cat([a * n + b, b * n + a, loop * n + loop])).values
    return key // n, key % n


def _relabelled(n, rows, cols, seed):
    """The graph with its 8-row windows in another order and the rows of each
    window too: other ids, and a block format of the same size."""
    g = _gen(seed)
    wins = torch.randperm(n // 8, generator=g, device="cuda")
    inner = torch.rand(n // 8, 8, generator=g, device="cuda").argsort(1)
    new = torch.cat([(wins[:, None] * 8 + inner).flatten(), torch.arange(n // 8 * 8, n, device="cuda")])
    key = torch.sort(new[rows] * n + new[cols]).values
    return key // n, key % n


def _rowptr(rows, n_pad):
    rp = torch.zeros(n_pad + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n_pad), 0)
    return rp


def _pad8(n):
    return n + 8 - n % 8  # the loaders' padding of the row count


def _uniform(shape, seed, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=_gen(seed), device="cuda") * (hi - lo) + lo


def _degree(rp, half):
    """rsqrt of the row lengths, 0 for the empty padding rows"""
    d = torch.rsqrt((rp[1:] - rp[:-1]).float())
    d = torch.where(torch.isfinite(d), d, torch.zeros_like(d))
    return d.half() if half else d


def _agg_features(case, seed):
    X = _uniform((case["n"], case["f"]), seed + 1)
    if case["dtype"] == "fp8":
        scale = X.abs().amax(1).clamp_min(1e-6) / 448.0
        return (X / scale[:, None]).to(torch.float8_e4m3fn), scale
    return X.to({"fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32}[case["dtype"]]), None


def _glorot(a, b, seed):
    lim = math.sqrt(6.0 / (a + b))
    return _uniform((a, b), seed, -lim, lim)


def _attention_features(case, seed):
    """X' = X W of an attention layer: uniform features projected, as the layer has them"""
    X = _uniform((case["n"], case["f"]), seed + 1)
    Xp = X @ _glorot(case["f"], case["f"], seed + 2)
    return Xp.to({"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}[case["dtype"]])


def _gat_weights(case, seed):
    h, f = case["heads"], case["f"]
    return (_glorot(case["fin"], h * f, seed + 2), _uniform((h, f), seed + 3, -0.4, 0.4),
            _uniform((h, f), seed + 4, -0.4, 0.4))


def _serve_sizes(case):
    g = torch.Generator()
    g.manual_seed(case["graphs"] + case["nmax"])
    u = torch.rand(case["graphs"], 2, generator=g).tolist()
    # node counts log-uniform from 1000, one of them the largest; mean degree 5 .. 50
    ns = [int(1000 * (case["nmax"] / 1000) ** a) for a, _ in u]
    ns[0] = case["nmax"]
    return [(n, 5.0 + 45.0 * b) for n, (_, b) in zip(ns, u)]


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "serve":
        jobs = []
        for i, (n, deg) in enumerate(_serve_sizes(case)):
            rows, cols = _graph(n, deg, seed * 64 + i)
            rp = _rowptr(rows, _pad8(n)).int()
            fmt = ops.block_convert(rp, cols.int(), _degree(rp, True), window=8, wide=8, part=32, n_cols=n)
            grp = serving.spmm_groups(fmt, m_out=n)
            part = torch.empty(max(grp.n_slots, 1) * 8 * case["f"], device="cuda")
            X = _uniform((n, case["f"]), seed * 64 + i + 1).half()
            jobs.append(serving.Job(fmt, grp, part, X, torch.empty(n, case["f"], device="cuda"), n))
        st["jobs"], st["batched"] = jobs, serving.BatchedSpmm(len(jobs))
        return st
    n = case["n"]
    # a conversion's outputs are as large as the graph makes them: one graph per case, relabelled
    rows, cols = _relabelled(n, *_graph(n, case["deg"], 1), seed) if kind == "convert" else _graph(n, case["deg"], seed)
    if kind == "agg":
        rp = _rowptr(rows, _pad8(n)).int()
        tf32, bf16 = case["dtype"] == "tf32", case["dtype"] == "bf16"
        st["fmt"] = ops.block_convert(rp, cols.int(), _degree(rp, not tf32), window=8, wide=4 if tf32 else 8, part=32,
                                      emit_empty=tf32, val_dtype=torch.bfloat16 if bf16 else None)
        st["X"], st["scale"] = _agg_features(case, seed)
    elif kind == "convert":
        st["rp"], st["col"] = _rowptr(rows, _pad8(n)).int(), cols.int()
        st["deg"] = _degree(st["rp"], True)
    elif kind == "gcn":
        st["info"] = layers.GCNInput(rows.cpu(), cols.cpu(), n)
        st["layer"] = layers.GCNConv(case["fin"], case["f"]).cuda()
        with torch.no_grad():
            st["layer"].weights.copy_(_glorot(case["fin"], case["f"], seed + 2))
        st["X"] = _uniform((n, case["fin"]), seed + 1).half().requires_grad_()
        st["dout"] = _uniform((n, case["f"]), seed + 5).half()
    elif kind == "attention":
        st["graph"] = gat.GATGraph(_rowptr(rows, n).int(), cols.int())
        st["X"] = _attention_features(case, seed)
    else:
        W, a0, a1 = _gat_weights(case, seed)
        st["X"] = _uniform((n, case["fin"]), seed + 1)
        st["dout"] = _uniform((n, case["heads"] * case["f"]), seed + 5)
        if kind == "gat":
            dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float16
            st["graph"] = gat.GATGraph(_rowptr(rows, n).int(), cols.int())
            st["graph"].transposed()
            layer = gat.GATConv(case["fin"], case["f"], case["heads"], HEADS_SLOPE, dt).cuda()
            with torch.no_grad():
                layer.W.copy_(W), layer.a0.copy_(a0), layer.a1.copy_(a1)
            st["X"] = st["X"].to(dt).requires_grad_()
            st["params"] = [layer.W, layer.a0, layer.a1]
        else:
            st["info"] = layers.GATInput(rows.cpu(), cols.cpu(), n)
            layer = layers.GATConv_multi(case["fin"], case["f"], 0.0, HEADS_SLOPE, case["heads"]).cuda()
            with torch.no_grad():
                layer.fc.weight.copy_(W.t())
                layer.a0.copy_(a0[:, None]), layer.a1.copy_(a1[:, None])
            st["X"] = st["X"].half().requires_grad_()
            st["dout"] = st["dout"].view(n, case["heads"], case["f"])
            st["params"] = [layer.fc.weight, layer.a0, layer.a1]
        st["layer"] = layer
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "agg":
        f = st["fmt"]
        if case["dtype"] in ("fp16", "tf32"):
            fn = SpMM_sr_bcrs.forward_fp16_gnn if case["dtype"] == "fp16" else SpMM_sr_bcrs.forward_tf32_gnn
            return fn(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, st["X"], f.n_rows, case["f"], case["n"])[0]
        return ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, st["X"], case["n"], x_scale=st["scale"])
    if kind == "convert":
        if case["form"] == "gcn":
            return Block_sr_bcrs.blockProcess_fp16_balance(st["rp"], st["col"], st["deg"], 8, 8, 32, device="cuda")
        return ATT_Block_v3.blockProcess_sddmm_balance_gnn_trans(st["rp"], st["col"], 8, 8, 32, device="cuda")
    if kind == "gcn":
        out = st["layer"](st["X"], st["info"])
        dX, dW = torch.autograd.grad(out, [st["X"], st["layer"].weights], st["dout"])
        return {"out": out.detach(), "dX": dX, "dW": dW}
    if kind == "attention":
        return st["graph"].attention(st["X"], slope=HEADS_SLOPE, stats=False)[0]
    if kind == "serve":
        st["batched"].run(st["jobs"])
        return [j.Y for j in st["jobs"]]
    out = st["layer"](st["X"], st["graph"] if kind == "gat" else st["info"])
    grads = torch.autograd.grad(out, [st["X"]] + st["params"], st["dout"].to(out.dtype))
    return {"out": out.detach(), "dX": grads[0], "dW": grads[1], "da0": grads[2], "da1": grads[3]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _agg_work(n, e, f, xs, vs, ys=4):
    """A padded condensed column per edge (its id and 8 window rows of values), X and Y once."""
    return {"bytes": e * (4 + 8 * vs) + n * f * (xs + ys), "flops": 2 * e * f}


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "serve":
        parts = [_agg_work(m, m * (d + 1), case["f"], 2, 2) for m, d in _serve_sizes(case)]
        return {k: int(sum(p[k] for p in parts)) for k in ("bytes", "flops")}
    e, f = n * (case["deg"] + 1), case.get("f", 0)
    if kind == "agg":
        xs, vs = {"fp16": (2, 2), "bf16": (2, 2), "fp8": (1, 2), "tf32": (4, 4)}[case["dtype"]]
        w = _agg_work(n, e, f, xs, vs)
    elif kind == "convert":
        per_col = 4 + (8 * 2 if case["form"] == "gcn" else 2 * 8 * 4)
        w = {"bytes": 8 * n + 4 * e + e * per_col, "flops": 0}
    elif kind == "gcn":
        fin, a = case["fin"], _agg_work(n, e, f, 2, 2, 2)
        w = {"bytes": 2 * a["bytes"] + 2 * n * (2 * fin + f), "flops": 2 * a["flops"] + 6 * n * fin * f}
    elif kind == "attention":
        xs = 4 if case["dtype"] == "fp32" else 2
        # structure and occupancy (a bit per slot), X' and the output once; logits and aggregation
        w = {"bytes": e * 5 + n * f * (xs + 4), "flops": 4 * e * f}
    else:
        hf, fin = case["heads"] * f, case["fin"]
        # forward and backward read the structure; X, X', the output and the incoming gradient once each way
        struct = e * 5 if kind == "gat" else e * 40
        w = {"bytes": 2 * struct + n * (2 * fin * 2 + 2 * hf * 2 + 2 * hf * 4),
             "flops": 6 * n * fin * hf + 6 * e * hf}
    return {k: int(v) for k, v in w.items()}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _values(rows, cols, deg, dtype):
    """Block values as the format holds them: the product of the degree factors rounded once."""
    return (deg[rows].float() * deg[cols].float()).to(dtype).double()


def _spmm64(rows, cols, vals, n, X):
    A = torch.sparse_csr_tensor(_rowptr(rows, n), cols, vals, (n, X.shape[0]), check_invariants=False)
    return A @ X.double()


def _softmax64(e, rows, n):
    m = torch.full((n,), -math.inf, dtype=torch.float64, device="cuda").scatter_reduce_(0, rows, e, "amax")
    p = torch.exp(e - m[rows])
    return p / torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, p)[rows]


def _gat64(case, seed, rows, cols, X, dout, round_w):
    """Additive attention layer and its gradients by autograd, one head at a time."""
    n, h, f = case["n"], case["heads"], case["f"]
    W, a0, a1 = (t.to(round_w).double().requires_grad_() for t in _gat_weights(case, seed))
    X = X.double().requires_grad_()
    outs, Xp = [], (X @ W).view(n, h, f)
    for k in range(h):
        x = Xp[:, k]
        e = torch.nn.functional.leaky_relu((x @ a0[k])[rows] + (x @ a1[k])[cols], HEADS_SLOPE)
        # the shift by the row maximum cancels in value and gradient
        m = torch.full((n,), -math.inf, dtype=torch.float64, device="cuda").scatter_reduce(0, rows, e.detach(), "amax")
        p = torch.exp(e - m[rows])
        s = torch.zeros(n, dtype=torch.float64, device="cuda").index_add(0, rows, p)
        outs.append(torch.zeros(n, f, dtype=torch.float64, device="cuda").index_add(0, rows, p[:, None] * x[cols])
                    / s[:, None])
    out = torch.stack(outs, 1)
    grads = torch.autograd.grad(out, [X, W, a0, a1], dout.double().view(n, h, f))
    return (out.detach(),) + grads


def exact(case, seed):
    kind = case["kind"]
    if kind == "convert":
        return None  # a format: ids, maps and values that the conversion must reproduce bit for bit
    if kind == "serve":
        ys = []
        for i, (n, deg) in enumerate(_serve_sizes(case)):
            rows, cols = _graph(n, deg, seed * 64 + i)
            vals = _values(rows, cols, _degree(_rowptr(rows, n), True), torch.float16)
            ys.append(_spmm64(rows, cols, vals, n, _uniform((n, case["f"]), seed * 64 + i + 1).half()))
        return ys
    n = case["n"]
    rows, cols = _graph(n, case["deg"], seed)
    if kind == "agg":
        tf32 = case["dtype"] == "tf32"
        vt = {"tf32": torch.float32, "bf16": torch.bfloat16}.get(case["dtype"], torch.float16)
        X, scale = _agg_features(case, seed)
        X = X.double() if scale is None else X.double() * scale.double()[:, None]
        return _spmm64(rows, cols, _values(rows, cols, _degree(_rowptr(rows, n), not tf32), vt), n, X)
    if kind == "gcn":
        vals = _values(rows, cols, _degree(_rowptr(rows, n), True), torch.float16)
        X = _uniform((n, case["fin"]), seed + 1).half().double()
        W = _glorot(case["fin"], case["f"], seed + 2).half().double()
        dXp = _spmm64(rows, cols, vals, n, _uniform((n, case["f"]), seed + 5).half())
        return {"out": _spmm64(rows, cols, vals, n, X @ W), "dX": dXp @ W.t(), "dW": X.t() @ dXp}
    if kind == "attention":
        X = _attention_features(case, seed).double()
        e = torch.cat([(X[r] * X[c]).sum(1) for r, c in zip(rows.split(1 << 21), cols.split(1 << 21))])
        p = _softmax64(torch.nn.functional.leaky_relu(e, HEADS_SLOPE), rows, n)
        return _spmm64(rows, cols, p, n, X)
    X = _uniform((n, case["fin"]), seed + 1)
    dout = _uniform((n, case["heads"] * case["f"]), seed + 5)
    dt = torch.bfloat16 if case.get("dtype") == "bf16" else torch.float16
    out, dX, dW, da0, da1 = _gat64(case, seed, rows, cols, X.to(dt), dout, torch.float32)
    if kind == "gat":
        return {"out": out.flatten(1), "dX": dX, "dW": dW, "da0": da0, "da1": da1}
    return {"out": out, "dX": dX, "dW": dW.t(), "da0": da0[:, None], "da1": da1[:, None]}

"""Performance cases of the sparse hot path: the calls that a user of this framework makes, over
the range of sizes, patterns, value types and directions that they are made with.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes
a case's inputs on the GPU, ``run`` makes one pass through the public entry points, ``work`` counts
the bytes and operations that a pass cannot do without, and ``exact`` computes a pass's outputs in
64 bits with plain torch.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import armsparse_gb300 as A
from armsparse_gb300 import gcn, selector

DEVICE = "cuda"
_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # The SpMV driver's matrix (density 0.01): the smallest call, where the launch and the
        # way to it are most of the time.
        {"name": "spmv_4096", "op": "spmv", "layout": "csr", "pattern": "uniform", "rows": 4096,
         "cols": 4096, "nnz": 167_772},
        # One aggregation of a citation-sized graph at an odd width (47 classes): a small call of
        # short rows and a few hubs whose rows of B fit no vector load.
        {"name": "spmm_f32_citation_n47", "op": "spmm", "dtype": "f32", "out": "f32",
         "pattern": "graph", "rows": 19_717, "cols": 19_717, "nnz": 108_365, "width": 47},
        # The SpMM driver's case: 4096 cubed at density 0.01, a wide dense operand.
        {"name": "spmm_f32_4096", "op": "spmm", "dtype": "f32", "out": "f32",
         "pattern": "uniform", "rows": 4096, "cols": 4096, "nnz": 167_772, "width": 4096},
        # bf16 storage in and out at a feature width that fills no whole tile (100 columns:
        # 200-byte rows).
        {"name": "spmm_bf16_100k_n100", "op": "spmm", "dtype": "bf16", "out": "bf16",
         "pattern": "uniform", "rows": 100_000, "cols": 100_000, "nnz": 2_000_000, "width": 100},
        # Skewed row lengths with the library's own (order-keeping) choice of kernels: hub rows
        # of up to nearly all columns beside rows of a few entries.
        {"name": "spmm_f32_powerlaw_n128", "op": "spmm", "dtype": "f32", "out": "f32",
         "pattern": "powerlaw", "rows": 300_000, "cols": 300_000, "nnz": 5_830_000, "width": 128},
        # Edge scores of a graph from fp32 node features (attention logits, edge gradients).
        {"name": "sddmm_f32_graph_k128", "op": "sddmm", "path": "simt", "pattern": "graph",
         "rows": 300_000, "cols": 300_000, "nnz": 6_000_000, "width": 128},
        # The SDDMM driver's case on the tensor cores: 4096 cubed at density 0.1.
        {"name": "sddmm_tc_4096", "op": "sddmm", "path": "tc", "pattern": "uniform",
         "rows": 4096, "cols": 4096, "nnz": 1_677_721, "width": 4096},
        # The transpose of a large skewed matrix with its values (once per graph, and per step
        # where the values change).
        {"name": "csr2csc_1m", "op": "csr2csc", "pattern": "powerlaw", "rows": 1_000_000,
         "cols": 1_000_000, "nnz": 16_800_000},
        # Sparse times sparse into a dense result, as the SpMM driver times it.
        {"name": "spgemm_4096", "op": "spgemm", "pattern": "uniform", "rows": 4096, "cols": 4096,
         "nnz": 167_772, "width": 4096},
        # A hidden layer of a large graph network, forward and backward, edge values trainable,
        # bf16 storage, the ReLU in the store: the largest call.
        {"name": "layer_bf16_2m_n256", "op": "layer", "dtype": "bf16", "pattern": "graph",
         "rows": 2_400_000, "cols": 2_400_000, "nnz": 35_800_000, "width": 256, "relu": True,
         "classes": 0},
        # The same network's head: 47 classes carried 48 wide, with the softmax cross-entropy,
        # forward and backward.
        {"name": "head_bf16_2m_n48", "op": "layer", "dtype": "bf16", "pattern": "graph",
         "rows": 2_400_000, "cols": 2_400_000, "nnz": 35_800_000, "width": 48, "relu": False,
         "classes": 47},
        # The citation network as a whole (500 sparse features, 64 hidden, 3 classes), forward
        # and backward: log-probabilities and the gradients of all weights.
        {"name": "net_citation", "op": "net", "pattern": "graph", "rows": 19_717,
         "cols": 19_717, "nnz": 108_365, "features": 500, "hidden": 64, "classes": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes over their logarithm, odd ones among them."""
    op = rng.choice(["spmv", "spmm", "spmm", "spmm", "reduce", "sddmm", "sddmm", "csr2csc",
                     "spgemm", "layer", "layer", "net"])
    if op == "spmv":
        rows = _log_int(rng, 1_000, 1_000_000)
        return {"op": op, "layout": rng.choice(["csr", "csr", "vcsr4"]),
                "pattern": rng.choice(["uniform", "powerlaw"]), "rows": rows, "cols": rows,
                "nnz": min(rows * _log_int(rng, 4, 60), rows * rows // 8)}
    if op in ("spmm", "reduce"):
        rows = _log_int(rng, 2_000, 400_000)
        nnz = min(rows * _log_int(rng, 4, 60), 6_000_000, rows * rows // 16)
        width = min(_log_int(rng, 8, 1024), max(8, 1_000_000_000 // nnz))
        if rng.random() < 0.6:  # most feature widths are multiples of eight
            width = max(8, width // 8 * 8)
        case = {"op": op, "pattern": rng.choice(["uniform", "powerlaw", "graph"]), "rows": rows,
                "cols": rows, "nnz": nnz + rows, "width": width}
        if op == "reduce":
            case["reduce"] = rng.choice(["sum", "max"])
        else:
            case["dtype"] = rng.choice(["f32", "f32", "bf16"])
            case["out"] = "f32" if case["dtype"] == "f32" else rng.choice(["f32", "bf16"])
        return case
    if op == "sddmm":
        path = rng.choice(["simt", "simt", "tc"])
        if path == "tc":  # patterns that fill the output tiles
            rows, cols = _log_int(rng, 500, 5_000), _log_int(rng, 500, 5_000)
            return {"op": op, "path": path, "pattern": "uniform", "rows": rows, "cols": cols,
                    "nnz": int(rows * cols * rng.uniform(0.02, 0.2)),
                    "width": _log_int(rng, 64, 4096)}
        rows = _log_int(rng, 2_000, 400_000)
        return {"op": op, "path": path, "pattern": rng.choice(["uniform", "graph"]),
                "rows": rows, "cols": rows,
                "nnz": min(rows * _log_int(rng, 4, 30), 6_000_000, rows * rows // 16) + rows,
                "width": max(16, _log_int(rng, 16, 512) // 4 * 4 + rng.choice([0, 0, 0, 1]))}
    if op == "csr2csc":
        rows, cols = _log_int(rng, 2_000, 1_500_000), _log_int(rng, 2_000, 1_500_000)
        return {"op": op, "pattern": rng.choice(["uniform", "powerlaw"]), "rows": rows,
                "cols": cols, "nnz": min(rows * _log_int(rng, 4, 30), 16_000_000,
                                         rows * cols // 16)}
    if op == "spgemm":
        rows = _log_int(rng, 500, 8_000)
        return {"op": op, "pattern": "uniform", "rows": rows, "cols": rows,
                "nnz": int(rows * rows * rng.uniform(0.002, 0.02)), "width": rows}
    if op == "layer":
        rows = _log_int(rng, 10_000, 1_000_000)
        classes = rng.choice([0, 0, rng.randint(3, 60)])
        width = (classes + 7) // 8 * 8 if classes else max(16, _log_int(rng, 16, 256) // 8 * 8)
        return {"op": op, "dtype": "bf16" if classes else rng.choice(["f32", "bf16"]),
                "pattern": "graph", "rows": rows, "cols": rows,
                "nnz": min(rows * _log_int(rng, 4, 25), 12_000_000) + rows, "width": width,
                "relu": not classes and rng.random() < 0.5, "classes": classes}
    rows = _log_int(rng, 2_000, 60_000)
    return {"op": "net", "pattern": "graph", "rows": rows, "cols": rows,
            "nnz": rows * _log_int(rng, 3, 20) + rows, "features": rng.randint(50, 600),
            "hidden": rng.choice([16, 32, 64, 128]), "classes": rng.randint(3, 20)}


# ---- inputs ---------------------------------------------------------------------------------
def _generator(seed, stream=0):
    return torch.Generator(device=DEVICE).manual_seed(seed * 16 + stream)


def _powerlaw_ids(n, exponent, u):
    """Indices 0..n-1 at the shares u in [0, 1) of weights that follow a power law (index 0 the
    heaviest), by its inverse: the same indices for the same u on every run."""
    s = 1 / (exponent - 1)  # weight of the quantile q, q from 0.5 / n to 1: q^-s
    lo = 0.5 / n
    if s == 1.0:
        q = lo ** (1 - u)
    else:
        q = (lo ** (1 - s) + u * (1 - lo ** (1 - s))) ** (1 / (1 - s))
    return (q * n).long().clamp_(0, n - 1)


def _pattern(case, gen):
    """(rowptr, colind) with exactly case["nnz"] distinct entries, columns ascending in a row.
    uniform: both indices uniform; powerlaw: row lengths follow a power law of exponent 2.0,
    columns uniform; graph: both ends follow one of exponent 2.1, self-loops on every node."""
    rows, cols, nnz, kind = case["rows"], case["cols"], case["nnz"], case["pattern"]
    rand = lambda m: torch.rand(m, generator=gen, device=DEVICE, dtype=torch.float64)
    loops = kind == "graph"
    want = nnz - rows if loops else nnz
    if kind != "uniform":
        exponent = 2.1 if loops else 2.0
        place = torch.randperm(rows, generator=gen, device=DEVICE)
    keys = torch.empty(0, dtype=torch.int64, device=DEVICE)
    factor = 1.1 if kind == "uniform" else 1.75
    while keys.numel() < want:
        m = int((want - keys.numel()) * factor) + 1024
        if kind == "uniform":
            new = torch.randint(0, rows * cols, (m,), generator=gen, device=DEVICE)
        else:
            r = place[_powerlaw_ids(rows, exponent, rand(m))]
            if loops:
                c = place[_powerlaw_ids(rows, exponent, rand(m))]
                r, c = r[r != c], c[r != c]
            else:
                c = torch.randint(0, cols, (m,), generator=gen, device=DEVICE)
            new = r * cols + c
        keys = torch.unique(torch.cat([keys, new]))
    if keys.numel() > want:
        keep = torch.randperm(keys.numel(), generator=gen, device=DEVICE)[:want]
        keys = keys[torch.sort(keep).values]
    if loops:
        ids = torch.arange(rows, device=DEVICE)
        keys = torch.sort(torch.cat([keys, ids * (cols + 1)])).values
    r = torch.div(keys, cols, rounding_mode="floor")
    rowptr = torch.zeros(rows + 1, dtype=torch.int64, device=DEVICE)
    rowptr[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    return rowptr.to(torch.int32), (keys - r * cols).to(torch.int32)


def _uniform(shape, gen, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, device=DEVICE) * (hi - lo) + lo


def _normal(shape, gen, dtype=torch.float32):
    out = torch.empty(shape, device=DEVICE, dtype=dtype)
    for lo in range(0, shape[0], 1 << 18):  # by blocks: no fp32 copy of a large bf16 operand
        hi = min(shape[0], lo + (1 << 18))
        out[lo:hi] = torch.randn((hi - lo, *shape[1:]), generator=gen, device=DEVICE)
    return out


def _inputs(case, seed):
    """The tensors that a case's call takes, from the seed alone."""
    op, gen = case["op"], _generator(seed)
    rowptr, colind = _pattern(case, gen)
    d = {"rowptr": rowptr, "colind": colind}
    nnz = colind.numel()
    if op in ("spmv", "spmm", "reduce", "csr2csc", "spgemm"):
        d["val"] = _uniform(nnz, gen)
    if op == "spmv":
        d["x"] = _uniform(case["cols"], gen)
    elif op in ("spmm", "reduce"):
        d["B"] = _uniform((case["cols"], case["width"]), gen)
        if op == "spmm":
            dtype = _DTYPES[case["dtype"]]
            d["val"], d["B"] = d["val"].to(dtype), d["B"].to(dtype)
    elif op == "spgemm":
        d["b_rowptr"], d["b_colind"] = _pattern(
            dict(case, rows=case["cols"], cols=case["width"]), gen)
        d["b_val"] = _uniform(d["b_colind"].numel(), gen)
    elif op == "sddmm":
        d["aval"] = _uniform(nnz, gen, 0.5, 1.5)
        d["X"] = _normal((case["rows"], case["width"]), gen)
        d["Y"] = _normal((case["cols"], case["width"]), gen)
    elif op == "layer":
        dtype = _DTYPES[case["dtype"]]
        deg = (rowptr[1:] - rowptr[:-1]).long()
        norm = torch.repeat_interleave(1 / deg.float().sqrt(), deg)
        d["w"] = norm * _uniform(nnz, gen, 0.5, 1.5)
        d["h"] = _normal((case["cols"], case["width"]), gen, dtype)
        if case["classes"]:
            d["h"][:, case["classes"]:] = 0  # the padding columns
            d["y"] = torch.randint(0, case["classes"], (case["rows"],), generator=gen,
                                   device=DEVICE)
        else:
            d["g"] = _normal((case["rows"], case["width"]), gen, dtype)
    elif op == "net":
        rows, feats, hidden, classes = (case[k] for k in ("rows", "features", "hidden", "classes"))
        x = _uniform((rows, feats), gen, 0.0, 1.0)
        d["x"] = torch.where(_uniform((rows, feats), gen, 0.0, 1.0) < 0.1, x, 0.0)
        d["val"] = torch.ones(nnz, device=DEVICE)
        d["y"] = torch.randint(0, classes, (rows,), generator=gen, device=DEVICE)
        train = torch.randperm(rows, generator=gen, device=DEVICE)[:60 * classes]
        d["train"] = torch.sort(train).values
        for i, (fan_in, fan_out) in enumerate(((feats, hidden), (hidden, classes)), 1):
            a = math.sqrt(6.0 / (fan_in + fan_out))
            d[f"W{i}"] = _uniform((fan_in, fan_out), gen, -a, a)
            d[f"b{i}"] = _uniform((fan_out,), gen, -0.1, 0.1)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    d["case"] = case
    op = case["op"]
    if op == "spmv" and case["layout"] == "vcsr4":
        d["v4"] = A.csr_to_vcsr4(d["rowptr"], d["colind"], d["val"])
    elif op == "layer":
        # the graph and its transpose, and the kernel that the selector names for the forward
        d["graph"] = gcn.Graph(d["rowptr"], d["colind"], d["w"], case["cols"])
        d["csc"], d["csc_pos"] = d["graph"].csc, d["graph"].csc_pos
        d["w"].requires_grad_(True)
        d["h"].requires_grad_(True)
        pick = selector.Selector.load().choose(d["rowptr"], case["cols"], case["width"],
                                               _DTYPES[case["dtype"]])
        d["variants"] = (pick, 0)
    elif op == "net":
        d["graph"] = gcn.Graph(d["rowptr"], d["colind"], d["val"])
        d["feats"] = gcn.SparseFeatures(d["x"])
        model = gcn.Net(case["features"], case["hidden"], case["classes"], dropout=0.0).to(DEVICE)
        with torch.no_grad():
            for i, conv in enumerate((model.conv1, model.conv2), 1):
                conv.weight.copy_(d[f"W{i}"])
                conv.bias.copy_(d[f"b{i}"])
        d["model"], d["params"] = model, list(model.parameters())
        d["y_train"] = d["y"].index_select(0, d["train"])
    return d


def run(d):
    case = d["case"]
    op = case["op"]
    if op == "spmv":
        if case["layout"] == "vcsr4":
            return A.spmv_vcsr4(*d["v4"], d["x"])
        return A.spmv(d["rowptr"], d["colind"], d["val"], d["x"])
    if op == "spmm":
        return A.spmm(d["rowptr"], d["colind"], d["val"], d["B"], out_dtype=_DTYPES[case["out"]])
    if op == "reduce":
        return A.spmm_reduce(d["rowptr"], d["colind"], d["B"], val=d["val"], op=case["reduce"])
    if op == "sddmm":
        return A.sddmm(d["rowptr"], d["colind"], d["X"], d["Y"], aval=d["aval"],
                       tensor_cores=case["path"] == "tc")
    if op == "csr2csc":
        return A.csr2csc(d["rowptr"], d["colind"], d["val"], case["cols"])
    if op == "spgemm":
        return A.spgemm_dense(d["rowptr"], d["colind"], d["val"], d["b_rowptr"], d["b_colind"],
                              d["b_val"], case["width"])
    if op == "layer":
        colptr, rowind, w_csc = d["csc"]
        out = gcn.SPMMFunction.apply(d["rowptr"], d["colind"], colptr, rowind, d["h"], d["w"],
                                     w_csc, d["variants"], d["csc_pos"], case["relu"])
        if not case["classes"]:
            return (out.detach(), *torch.autograd.grad(out, (d["h"], d["w"]), d["g"]))
        loss = gcn.SoftmaxXent.apply(out, d["y"], case["classes"])
        return (out.detach(), loss.detach(), *torch.autograd.grad(loss, (d["h"], d["w"])))
    logp = d["model"](d["feats"], d["graph"])
    loss = F.nll_loss(logp.index_select(0, d["train"]), d["y_train"])
    return (logp.detach(), *torch.autograd.grad(loss, d["params"]))


def work(case):
    op, m, k, nnz = case["op"], case["rows"], case["cols"], case["nnz"]
    n = case.get("width", 1)
    index = 4 * (m + 1) + 4 * nnz
    if op == "spmv":
        return {"bytes": index + 4 * nnz + 4 * k + 4 * m, "flops": 2 * nnz}
    if op in ("spmm", "reduce"):
        size = 2 if case.get("dtype") == "bf16" else 4
        out = 2 if case.get("out") == "bf16" else 4
        return {"bytes": index + size * (nnz + k * n) + out * m * n, "flops": 2 * nnz * n}
    if op == "sddmm":
        return {"bytes": index + 8 * nnz + 4 * (m + k) * n, "flops": 2 * nnz * n}
    if op == "csr2csc":
        return {"bytes": index + 4 * nnz + 4 * (k + 1) + 8 * nnz, "flops": 0}
    if op == "spgemm":
        return {"bytes": 2 * (index + 4 * nnz) + 4 * m * n, "flops": 2 * nnz * nnz // k}
    if op == "layer":
        size = 2 if case["dtype"] == "bf16" else 4
        # the CSR and the CSC with their values, the permutation and the edge gradient; the
        # features in and out and the gradients in and out (the loss's stays inside)
        dense = 4 if not case["classes"] else 3
        return {"bytes": 2 * (index + 4 * nnz) + 8 * nnz + dense * size * m * n +
                8 * m * bool(case["classes"]), "flops": 6 * nnz * n}
    f, h, c = case["features"], case["hidden"], case["classes"]
    feats = m * f // 10  # stored features
    return {"bytes": 2 * (2 * index) + 2 * 8 * feats + 4 * 2 * (f * h + h * c) + 4 * m * c,
            "flops": 4 * (feats * h + nnz * (h + c)) + 6 * m * h * c}


# ---- the same in 64 bits --------------------------------------------------------------------
def _matrix64(rowptr, colind, val, n_cols):
    return torch.sparse_csr_tensor(rowptr.long(), colind.long(), val.double(),
                                   size=(rowptr.numel() - 1, n_cols))


def _row_ids(rowptr):
    deg = (rowptr[1:] - rowptr[:-1]).long()
    return torch.repeat_interleave(torch.arange(deg.numel(), device=deg.device), deg)


def _dots64(rows, cols, X, Y):
    """<X[rows[e]], Y[cols[e]]> per entry, by blocks of entries."""
    out = torch.empty(rows.numel(), dtype=torch.float64, device=rows.device)
    step = max(1, (1 << 28) // X.shape[1])
    for lo in range(0, rows.numel(), step):
        r, c = rows[lo:lo + step], cols[lo:lo + step]
        out[lo:lo + step] = (X[r].double() * Y[c].double()).sum(1)
    return out


def _transposed(rows, colind, val, n_rows, n_cols):
    order = torch.sort(colind, stable=True).indices
    colptr = torch.zeros(n_cols + 1, dtype=torch.int64, device=colind.device)
    colptr[1:] = torch.cumsum(torch.bincount(colind, minlength=n_cols), 0)
    return colptr, rows[order], val[order]


def _exact_net(d, case):
    params = [d[k].double().requires_grad_(True) for k in ("W1", "b1", "W2", "b2")]
    W1, b1, W2, b2 = params
    rows, cols = _row_ids(d["rowptr"]), d["colind"].long()
    in_norm = torch.bincount(rows, minlength=case["rows"]).double().rsqrt()[:, None]
    out_norm = torch.bincount(cols, minlength=case["rows"]).double().rsqrt()[:, None]

    def conv(x, W, b):
        z = (x @ W) * out_norm
        return torch.zeros_like(z).index_add(0, rows, z[cols]) * in_norm + b

    logp = F.log_softmax(conv(torch.relu(conv(d["x"].double(), W1, b1)), W2, b2), dim=1)
    loss = F.nll_loss(logp[d["train"]], d["y"][d["train"]])
    grads = torch.autograd.grad(loss, params)
    return (logp.detach(), *grads)


def exact(case, seed):
    d = _inputs(case, seed)
    op, m, k = case["op"], case["rows"], case["cols"]
    rows, cols = _row_ids(d["rowptr"]), d["colind"].long()
    if op == "spmv":
        return (_matrix64(d["rowptr"], cols, d["val"], k) @ d["x"].double()[:, None])[:, 0]
    if op == "spmm":
        return _matrix64(d["rowptr"], cols, d["val"], k) @ d["B"].double()
    if op == "reduce":
        out = torch.zeros(m, case["width"], dtype=torch.float64, device=DEVICE)
        step = max(1, (1 << 24) // m)  # columns at a time
        for lo in range(0, case["width"], step):
            part = d["val"].double()[:, None] * d["B"][:, lo:lo + step].double()[cols]
            if case["reduce"] == "sum":
                out[:, lo:lo + step].index_add_(0, rows, part)
            else:
                out[:, lo:lo + step] = out[:, lo:lo + step].index_reduce(
                    0, rows, part, "amax", include_self=False)
        return out
    if op == "sddmm":
        return d["aval"].double() * _dots64(rows, cols, d["X"], d["Y"])
    if op == "csr2csc":
        colptr, rowind, val = _transposed(rows, cols, d["val"], m, k)
        return colptr.to(torch.int32), rowind.to(torch.int32), val.double()
    if op == "spgemm":
        dense_b = _matrix64(d["b_rowptr"], d["b_colind"], d["b_val"], case["width"]).to_dense()
        return _matrix64(d["rowptr"], cols, d["val"], k) @ dense_b
    if op == "net":
        return _exact_net(d, case)
    out = _matrix64(d["rowptr"], cols, d["w"], k) @ d["h"].double()
    if case["classes"]:
        # scores, mean cross-entropy over the classes, gradients of the features and the edges
        logp = F.log_softmax(out[:, :case["classes"]], dim=1)
        loss = F.nll_loss(logp, d["y"])
        g = torch.zeros_like(out)
        g[:, :case["classes"]] = logp.exp()
        g[torch.arange(m, device=DEVICE), d["y"]] -= 1
        g /= m
        outs = (out, loss)
    else:
        g = d["g"].double()
        if case["relu"]:
            out = torch.relu(out)
            g = g * (out > 0)
        outs = (out,)
    colptr, rowind, w_csc = _transposed(rows, cols, d["w"], m, k)
    dh = _matrix64(colptr, rowind, w_csc, m) @ g
    return (*outs, dh, _dots64(rows, cols, g, d["h"]))

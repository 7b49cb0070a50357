"""The work that users of this package have it do, as cases that can be timed.

Each case is one call (or one training or solver step) through the public
entry points, at sizes from the package's own benchmark configurations and
tests or of the same kinds of matrix:

  zipf      rows of min(50000, ceil(s Z)) nonzeros, Z ~ Zipf(2): power-law matrices
  poisson   rows of max(1, Poisson(mean)) nonzeros at uniform columns
  stencil   the 5-point stencil on a square grid: PDE operators, local columns
  uniform   a fixed number of nonzeros anywhere: row lengths close to Poisson's
  chunglu   a symmetric Chung-Lu graph (exponent 2.5), values 1/sqrt(d_i d_j)

Patterns whose nonzeros are an output (SDDMM, gradients) have as many for
every seed.

``listed()`` holds the cases, ``draw(rng)`` gives another of the same ranges,
``prepare`` makes a user program's state on the GPU from a seed, ``run`` is one
pass, ``exact`` the same outputs in float64 from plain torch.
"""

import math

import numpy as np
import torch

import flagsparse_b200 as fs

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32, "float64": torch.float64}
BYTES = {"float16": 2, "bfloat16": 2, "float32": 4, "float64": 8}
ZIPF_CAP = 50_000


def listed():
    return [
        # one product with a small matrix inside a larger loop: launch latency
        {"name": "spmv small f32", "op": "spmv", "matrix": "poisson", "rows": 4096, "mean": 16.0, "dtype": "float32",
         "index": "int32"},
        # the package's headline: a large power-law matrix times a vector (ranking, graph analytics)
        {"name": "spmv powerlaw f32", "op": "spmv", "matrix": "zipf", "rows": 2_000_000, "mean": 20.0,
         "dtype": "float32", "index": "int32"},
        # the product of an iterative PDE solver: float64, short local rows, torch's int64 columns
        {"name": "spmv stencil f64", "op": "spmv", "matrix": "stencil", "rows": 1021 * 1021, "mean": 5.0,
         "dtype": "float64", "index": "int64"},
        # feature propagation over a large power-law matrix, fp32
        {"name": "spmm powerlaw f32 128", "op": "spmm", "matrix": "zipf", "rows": 1_000_000, "mean": 32.0,
         "dtype": "float32", "n": 128},
        # the same in mixed precision: bf16 values and features, fp32 sums
        {"name": "spmm powerlaw bf16 128", "op": "spmm", "matrix": "zipf", "rows": 1_000_000, "mean": 32.0,
         "dtype": "bfloat16", "n": 128},
        # the last layer of a node classifier: as many columns as classes, an odd width
        {"name": "spmm graph f32 47", "op": "spmm", "matrix": "chunglu", "rows": 170_001, "mean": 14.0,
         "dtype": "float32", "n": 47},
        # the unprepared call: checks, plan and product for a matrix that is used once
        {"name": "spmm once f32 16", "op": "spmm_once", "matrix": "poisson", "rows": 20_000, "mean": 24.0,
         "dtype": "float32", "n": 16},
        # edge scores of a graph: SDDMM on the adjacency's pattern
        {"name": "sddmm graph f32 64", "op": "sddmm", "matrix": "chunglu", "rows": 500_000, "mean": 25.0,
         "dtype": "float32", "n": 64},
        # a training step of a graph layer, forward and backward, mixed precision
        {"name": "train graph bf16 128", "op": "train", "matrix": "chunglu", "rows": 500_000, "mean": 25.0,
         "dtype": "bfloat16", "n": 128},
        # the same in fp32 on a small graph: launches and autograd around short kernels
        {"name": "train small f32 64", "op": "train", "matrix": "chunglu", "rows": 20_011, "mean": 25.0,
         "dtype": "float32", "n": 64},
        # many uneven systems at once: stencils and random matrices, SpMV and a 16-column SpMM, one graph launch
        {"name": "batched 256 f32 16", "op": "batched", "count": 256, "lo": 1_000, "hi": 200_000, "mean": 24.0,
         "dtype": "float32", "n": 16},
        # block-sparse weights: 16 x 16 blocks on the tensor cores
        {"name": "bsr16 bf16 128", "op": "bsr16", "block_rows": 65_536, "per_row": 8, "dtype": "bfloat16", "n": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, widths aligned and odd."""
    op = rng.choice(["spmv", "spmv", "spmm", "spmm", "spmm_once", "sddmm", "train", "batched", "bsr16"])
    if op == "batched":
        lo = _log_int(rng, 500, 5_000)
        return {"op": op, "count": _log_int(rng, 8, 200), "lo": lo, "hi": lo * rng.randint(5, 30),
                "mean": round(rng.uniform(8.0, 32.0), 2), "dtype": "float32", "n": rng.choice([8, 16, 32])}
    if op == "bsr16":
        return {"op": op, "block_rows": _log_int(rng, 500, 60_000), "per_row": rng.randint(2, 8),
                "dtype": rng.choice(["bfloat16", "float16"]), "n": rng.choice([64, 128])}
    matrix = rng.choice({"spmv": ["zipf", "poisson", "stencil"], "spmm": ["zipf", "poisson", "chunglu"],
                         "spmm_once": ["zipf", "poisson"], "sddmm": ["chunglu", "uniform"],
                         "train": ["chunglu"]}[op])
    mean = 5.0 if matrix == "stencil" else round(rng.uniform(6.0, 32.0), 2)
    case = {"op": op, "matrix": matrix, "mean": mean}
    if op == "spmv":
        rows = _log_int(rng, 3_000, 1_500_000)
        case["rows"] = round(math.sqrt(rows)) ** 2 if matrix == "stencil" else rows
        case["dtype"] = rng.choice(["float32", "float32", "float64", "bfloat16"])
        case["index"] = rng.choice(["int32", "int64"])
        return case
    case["rows"] = _log_int(rng, 3_000, 100_000 if op == "spmm_once" else 600_000)
    if op == "sddmm":
        case["dtype"] = rng.choice(["float32", "float32", "float64"])
        case["n"] = rng.choice([8, 16, 32, 64, 128, rng.randint(5, 130)])
    elif op == "spmm_once":
        case["dtype"] = "float32"
        case["n"] = rng.choice([8, 16, 64, rng.randint(3, 100)])
    else:
        case["dtype"] = rng.choice(["float32", "float32", "bfloat16", "bfloat16", "float16"])
        case["n"] = rng.choice([16, 32, 64, 128, rng.randint(5, 130)])
    return case


# ---------------------------------------------------------------- matrices

def _zipf_table(mean):
    """(cumulative probabilities, lengths) of ceil(s Z) for Z = 1 .. 50000 with P(Z) ~ Z^-2."""
    k = np.arange(1, ZIPF_CAP + 1, dtype=np.float64)
    p = k ** -2.0
    p /= p.sum()
    return np.cumsum(p), np.minimum(ZIPF_CAP, np.ceil(mean / 6.93 * k)), p



def _mean_nnz(matrix, rows, mean):
    """Expected nonzeros (repeated columns, which the generators merge, aside)."""
    if matrix == "poisson":
        return rows * (mean + math.exp(-mean))
    if matrix == "zipf":
        _, length, p = _zipf_table(mean)
        return rows * float((np.minimum(length, rows // 2) * p).sum())
    if matrix == "stencil":
        side = int(round(math.sqrt(rows)))
        return 5.0 * side * side - 4.0 * side
    return round(rows * mean) if matrix == "uniform" else 2.0 * round(rows * mean / 2.0)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _csr_of_keys(key, rows, cols):
    """indptr int64 and sorted int32 columns of the distinct keys row * cols + col."""
    key = torch.unique(key)
    r = key // cols
    indptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(r, minlength=rows), 0, out=indptr[1:])
    return indptr, (key - r * cols).to(torch.int32)


def _exactly(some, count, g):
    """`count` distinct keys out of those that some(m) draws."""
    key = torch.unique(some(count + count // 4))
    while key.numel() < count:
        key = torch.unique(torch.cat([key, some(count // 2 + 16)]))
    return key[torch.randperm(key.numel(), device="cuda", generator=g)[:count]]


def _pattern(matrix, rows, mean, g):
    """(indptr int64, columns int32, values float64 or None) of a square matrix on the GPU."""
    if matrix == "stencil":
        side = int(round(math.sqrt(rows)))
        i = torch.arange(rows, device="cuda")
        keys = []
        for di, dj in ((-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)):
            ok = ((i // side + di >= 0) & (i // side + di < side) & (i % side + dj >= 0) & (i % side + dj < side))
            keys.append(i[ok] * rows + i[ok] + di * side + dj)
        return (*_csr_of_keys(torch.cat(keys), rows, rows), None)
    if matrix == "chunglu":
        w = torch.arange(1, rows + 1, dtype=torch.float64, device="cuda") ** (-1.0 / 1.5)
        cum = torch.cumsum(w / w.sum(), 0)

        def edges(m):
            ends = torch.searchsorted(cum, torch.rand(2, m, dtype=torch.float64, device="cuda", generator=g))
            lo, hi = ends.clamp_(max=rows - 1).sort(0).values
            return (lo * rows + hi)[lo != hi]

        key = _exactly(edges, int(round(rows * mean / 2.0)), g)
        indptr, cols = _csr_of_keys(torch.cat([key, key % rows * rows + key // rows]), rows, rows)
        deg = (indptr[1:] - indptr[:-1]).double()
        vals = torch.rsqrt(torch.repeat_interleave(deg, indptr[1:] - indptr[:-1]) * deg[cols.long()])
        return indptr, cols, vals
    if matrix == "uniform":
        key = _exactly(lambda m: torch.randint(0, rows * rows, (m,), device="cuda", generator=g),
                       int(round(rows * mean)), g)
        return (*_csr_of_keys(key, rows, rows), None)
    if matrix == "poisson":
        rate = torch.full((rows,), mean, device="cuda")
        length = torch.poisson(rate, generator=g).long().clamp_(1, rows)
    else:
        cum, length, _ = _zipf_table(mean)
        z = torch.searchsorted(torch.from_numpy(cum).cuda(), torch.rand(rows, dtype=torch.float64, device="cuda",
                                                                          generator=g))
        length = torch.from_numpy(length).cuda()[z.clamp_(max=ZIPF_CAP - 1)].long().clamp_(max=rows // 2)
    r = torch.repeat_interleave(torch.arange(rows, device="cuda"), length)
    c = torch.randint(0, rows, (r.numel(),), device="cuda", generator=g)
    return (*_csr_of_keys(r * rows + c, rows, rows), None)


def _uniform(shape, g):
    return torch.rand(shape, dtype=torch.float32, device="cuda", generator=g) * 2 - 1


def _normal(shape, g):
    return torch.randn(shape, dtype=torch.float32, device="cuda", generator=g)


def _matrix(case, g):
    indptr, cols, vals = _pattern(case["matrix"], case["rows"], case["mean"], g)
    dt = DTYPES[case["dtype"]]
    if vals is None:
        if case["matrix"] == "stencil":  # a variable-coefficient operator: dominant diagonal, couplings near -1
            r = torch.repeat_interleave(torch.arange(case["rows"], device="cuda"), indptr[1:] - indptr[:-1])
            vals = torch.where(cols == r, 4.0, -1.0) * (1 + 0.1 * _uniform(cols.numel(), g))
        else:
            vals = _uniform(cols.numel(), g) if case["op"] == "spmv" else _normal(cols.numel(), g)
    return indptr, cols, vals.to(dt)


def _inputs(case, seed):
    g = _generator(seed)
    dt = DTYPES[case["dtype"]]
    if case["op"] == "bsr16":
        nb, per = case["block_rows"], case["per_row"]
        r = torch.arange(nb, device="cuda").repeat_interleave(per)
        key = r * nb + torch.randint(0, nb, (nb * per,), device="cuda", generator=g)
        indptr, cols = _csr_of_keys(key, nb, nb)
        return {"indptr": indptr, "indices": cols, "blocks": _normal((cols.numel(), 16, 16), g).to(dt),
                "B": _normal((nb * 16, case["n"]), g).to(dt)}
    if case["op"] == "batched":
        order = torch.randperm(case["count"], device="cuda", generator=g).tolist()
        mats = []
        for k in order:
            rows = _batch_rows(case, k)
            kind = "stencil" if k % 2 == 0 else "poisson"
            one = dict(case, op="spmv", matrix=kind, rows=rows)
            indptr, cols, vals = _matrix(one, g)
            mats.append({"indptr": indptr, "indices": cols, "data": vals, "x": _uniform(rows, g),
                         "B": _uniform((rows, case["n"]), g)})
        return {"mats": mats}
    indptr, cols, vals = _matrix(case, g)
    d = {"indptr": indptr, "indices": cols, "data": vals}
    m = case["rows"]
    if case["op"] == "spmv":
        d["x"] = _uniform(m, g).to(dt)
        if case["index"] == "int64":
            d["indices"] = cols.to(torch.int64)
    elif case["op"] == "sddmm":
        d["x"], d["y"] = _normal((m, case["n"]), g).to(dt), _normal((m, case["n"]), g).to(dt)
    else:
        d["B"] = _normal((m, case["n"]), g).to(dt)
        if case["op"] == "train":
            d["dY"] = _normal((m, case["n"]), g).to(dt)
    return d


def _batch_rows(case, k):
    """Row counts spread evenly over the logarithm of [lo, hi]; squares for the stencils (even k)."""
    rows = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((k + 0.5) / case["count"])))
    return max(2, int(round(math.sqrt(rows)))) ** 2 if k % 2 == 0 else rows


# ---------------------------------------------------------------- one pass

def prepare(case, seed):
    d = _inputs(case, seed)
    op, m = case["op"], case.get("rows")
    if op == "spmv":
        return {"op": op, "x": d["x"], "p": fs.prepare_spmv_csr(d["data"], d["indices"], d["indptr"], (m, m))}
    if op == "spmm":
        return {"op": op, "B": d["B"], "p": fs.prepare_spmm_csr_route(d["data"], d["indices"], d["indptr"], (m, m))}
    if op == "spmm_once":
        return {"op": op, "shape": (m, m), **d}
    if op == "sddmm":
        return {"op": op, "x": d["x"], "y": d["y"],
                "p": fs.prepare_sddmm_csr(d["indices"], d["indptr"], (m, m), k_hint=case["n"])}
    if op == "train":
        return {"op": op, "dY": d["dY"], "vals": d["data"].requires_grad_(True), "X": d["B"].requires_grad_(True),
                "p": fs.prepare_spmm_csr_autograd(d["data"].detach(), d["indices"], d["indptr"], (m, m))}
    if op == "batched":
        b = fs.BatchedCsr([(q["data"], q["indices"], q["indptr"], (q["x"].numel(), q["x"].numel()))
                           for q in d["mats"]], n_dense=case["n"])
        for i, q in enumerate(d["mats"]):
            b.x_view(i).copy_(q["x"])
            b.B_view(i).copy_(q["B"])
        b.tune()
        b.capture()
        return {"op": op, "b": b}
    size = case["block_rows"] * 16
    return {"op": op, "B": d["B"], "p": fs.prepare_spmm_bsr16(d["blocks"], d["indices"], d["indptr"], (size, size))}


def run(state):
    op = state["op"]
    if op == "spmv":
        return fs.flagsparse_spmv_csr(x=state["x"], prepared=state["p"])
    if op == "spmm":
        return fs.flagsparse_spmm_csr_run(state["p"], state["B"])
    if op == "spmm_once":
        return fs.flagsparse_spmm_csr(state["data"], state["indices"], state["indptr"], state["B"], state["shape"])
    if op == "sddmm":
        return fs.flagsparse_sddmm_csr(x=state["x"], y=state["y"], prepared=state["p"])
    if op == "train":
        Y = fs.flagsparse_spmm_csr_autograd(state["vals"], state["X"], prepared=state["p"])
        dvals, dX = torch.autograd.grad(Y, (state["vals"], state["X"]), state["dY"])
        return {"Y": Y, "dX": dX, "dvals": dvals}
    if op == "batched":
        y, C = state["b"].run()
        return {"y": y, "C": C}
    return fs.flagsparse_spmm_bsr16(B=state["B"], prepared=state["p"])


# ---------------------------------------------------------------- work and exactness

def work(case):
    s, op = BYTES[case["dtype"]], case["op"]
    if op == "bsr16":
        nb, n = case["block_rows"], case["n"]
        nnzb = nb * case["per_row"]
        return {"bytes": nnzb * (256 * s + 4) + (nb + 1) * 8 + 2 * nb * 16 * n * s, "flops": 2 * nnzb * 256 * n}
    if op == "batched":
        n, nnz, rows = case["n"], 0.0, 0
        for k in range(case["count"]):
            r = _batch_rows(case, k)
            nnz += _mean_nnz("stencil" if k % 2 == 0 else "poisson", r, case["mean"])
            rows += r
        return {"bytes": nnz * (s + 4) + (rows + 1) * 8 + 2 * rows * (n + 1) * s, "flops": 2 * nnz * (n + 1)}
    m = case["rows"]
    nnz = _mean_nnz(case["matrix"], m, case["mean"])
    if op == "spmv":
        return {"bytes": nnz * (s + (8 if case["index"] == "int64" else 4)) + (m + 1) * 8 + 2 * m * s,
                "flops": 2 * nnz}
    n = case["n"]
    if op == "sddmm":  # pattern, both operands, one value out per nonzero
        return {"bytes": nnz * (4 + s) + (m + 1) * 8 + 2 * m * n * s, "flops": 2 * nnz * n}
    if op == "train":  # pattern, values and their gradient; X, dY, Y, dX
        return {"bytes": nnz * (4 + 2 * s) + (m + 1) * 8 + 4 * m * n * s, "flops": 6 * nnz * n}
    return {"bytes": nnz * (4 + s) + (m + 1) * 8 + 2 * m * n * s, "flops": 2 * nnz * n}


def tolerance(case):
    """About four times what the same sums in another order differ by (plain torch sums at the
    working precision, long rows among them); in 16 bits, values that round the other way."""
    return {"float64": {"rel": 6e-15, "max": 1.5e-13}, "float32": {"rel": 5e-6, "max": 1.2e-3},
            "float16": {"rel": 1.2e-4, "max": 2e-3}, "bfloat16": {"rel": 1e-3, "max": 1.6e-2}}[case["dtype"]]


def _rows_of(indptr):
    return torch.repeat_interleave(torch.arange(indptr.numel() - 1, device="cuda"), indptr[1:] - indptr[:-1])


def _product(rows, cols, vals, B, m):
    """sum over nonzeros of vals * B[cols] into m rows, float64, in parts that fit."""
    B = B.double()
    out = torch.zeros((m, *B.shape[1:]), dtype=torch.float64, device="cuda")
    width = B.shape[1] if B.ndim == 2 else 1
    step = max(1, (1 << 28) // width)
    for at in range(0, cols.numel(), step):
        part = slice(at, at + step)
        v = vals[part].double()
        out.index_add_(0, rows[part], (v[:, None] if B.ndim == 2 else v) * B[cols[part].long()])
    return out


def _dots(rows, cols, x, y):
    out = torch.empty(cols.numel(), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // x.shape[1])
    for at in range(0, cols.numel(), step):
        part = slice(at, at + step)
        out[part] = (x[rows[part]].double() * y[cols[part].long()].double()).sum(1)
    return out


def exact(case, seed):
    d = _inputs(case, seed)
    op = case["op"]
    if op == "bsr16":
        B = d["B"].double().view(-1, 16, case["n"])
        rows = _rows_of(d["indptr"])
        out = torch.zeros_like(B)
        for at in range(0, rows.numel(), 32768):
            part = slice(at, at + 32768)
            out.index_add_(0, rows[part], torch.bmm(d["blocks"][part].double(), B[d["indices"][part].long()]))
        return out.view(-1, case["n"])
    if op == "batched":
        ys, Cs = [], []
        for q in d["mats"]:
            rows = _rows_of(q["indptr"])
            ys.append(_product(rows, q["indices"], q["data"], q["x"], q["x"].numel()))
            Cs.append(_product(rows, q["indices"], q["data"], q["B"], q["x"].numel()))
        return {"y": torch.cat(ys), "C": torch.cat(Cs)}
    rows = _rows_of(d["indptr"])
    if op == "spmv":
        return _product(rows, d["indices"], d["data"], d["x"], case["rows"])
    if op == "sddmm":
        return _dots(rows, d["indices"], d["x"], d["y"])
    Y = _product(rows, d["indices"], d["data"], d["B"], case["rows"])
    if op != "train":
        return Y
    return {"Y": Y, "dX": _product(d["indices"].long(), rows, d["data"], d["dY"], case["rows"]),
            "dvals": _dots(rows, d["indices"], d["dY"], d["B"])}

"""Performance cases of the library: what a program does with it, through its public entry points.

Each case is one call (or one training step) that callers make in earnest: single products of
every storage format, from the 100000-row matrix of the CPU-sized configuration to matrices
far larger than L2; products with many vectors or many matrices; PageRank in the reference's
mode, in mixed precision, batched over seed sets, and differentiated.  ``listed`` gives the
fixed cases, ``draw`` others of the same ranges, ``prepare`` what a program holds before the
call, ``run`` one pass, ``work`` the bytes and operations it cannot do without and ``exact``
its result in 64-bit arithmetic from plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tbsla_gb300 import autograd, capi

STORE = {"f64": capi.F64, "f32": capi.F32, "bf16": capi.BF16}
STORE_BIT = {"f64": capi.STORE_F64, "f32": capi.STORE_F32, "bf16": capi.STORE_BF16}
VALUE_BYTES = {"f64": 8, "f32": 4, "bf16": 2}
TORCH = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}


def vector_dtype(store):
    """The vectors that go with a value store: FP64 for F64, FP32 for F32 and BF16."""
    return torch.float64 if store == "f64" else torch.float32


def listed():
    return [
        # the smallest products: the configuration the reference's CPU path is timed on (n = 1e5,
        # c = 10, in L2); latency and launches count
        {"name": "spmv_csr_f64_small", "kind": "spmv", "fmt": "CSR", "store": "f64", "n": 100_000, "c": 10},
        # the memory-bound product of the headline's shape (c = 16), eight times L2
        {"name": "spmv_csr_f64_large", "kind": "spmv", "fmt": "CSR", "store": "f64", "n": 1 << 22, "c": 16},
        # ragged rows (log-normal lengths, empty rows, a few hubs), half band and half scattered
        # columns: meshes with refinement, term-document matrices; single precision, odd sizes
        {"name": "spmv_coo_f32_ragged", "kind": "ragged", "fmt": "COO", "store": "f32", "n": 600_011, "mean": 14},
        # the drop-in classes' own call: host vectors in and out, r = A (A x + x)
        {"name": "axpx_host_ell_f64", "kind": "axpx_host", "fmt": "ELL", "store": "f64", "n": 1_000_003, "c": 9},
        # many right-hand sides through one matrix (block solvers, graph features)
        {"name": "spmm_csr_f32_k32", "kind": "spmm", "store": "f32", "n": 1 << 20, "c": 16, "k": 32},
        # DENSE format product in single precision, ragged sizes
        {"name": "gemv_dense_f32", "kind": "dense", "store": "f32", "rows": 8_000, "cols": 9_001, "k": 1},
        # many uneven matrices in one launch (ensembles, block-diagonal problems)
        {"name": "batch_f32_64", "kind": "batch", "store": "f32", "count": 64, "n_max": 100_000},
        # Matrix::page_rank as the reference's driver calls it on its own column-stochastic matrix
        {"name": "pagerank_reference", "kind": "pagerank", "graph": "cqmat", "n": 100_000, "c": 10,
         "mode": "reference", "precision": "f64", "accel": 0},
        # web-graph PageRank to 1e-12 in mixed precision with accelerated corrections
        {"name": "pagerank_rmat_f32", "kind": "pagerank", "graph": "rmat", "scale": 21, "mode": "dangling",
         "precision": "f32", "accel": 1},
        # personalized PageRank of many seed sets (recommendation, local clustering)
        {"name": "ppr_batched_f32_k64", "kind": "ppr", "scale": 17, "k": 64, "precision": "f32", "refined": True,
         "accel": 1},
        # one training step on edge weights through the PageRank fixed point: forward and adjoint solve
        {"name": "pagerank_grad_rmat", "kind": "pagerank_grad", "scale": 16},
        # one training step on a sparse layer's weights: forward, dL/dvalues, dL/dx
        {"name": "spmv_grad_f32", "kind": "spmv_grad", "store": "f32", "n": 1 << 20, "c": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "ragged", "axpx_host", "spmm", "dense", "batch", "pagerank", "pagerank",
                       "ppr", "pagerank_grad", "spmv_grad"])
    store = rng.choice(["f64", "f32", "bf16"])
    if kind == "spmv":
        n = _log(rng, 1_000, 3_500_000)
        return {"kind": kind, "fmt": rng.choice(["CSR", "ELL", "COO"]), "store": store, "n": n,
                "c": rng.randint(2, 18)}
    if kind == "ragged":
        return {"kind": kind, "fmt": rng.choice(["CSR", "COO"]), "store": store, "n": _log(rng, 2_000, 1_500_000),
                "mean": rng.randint(4, 40)}
    if kind == "axpx_host":
        return {"kind": kind, "fmt": rng.choice(["CSR", "ELL", "COO"]), "store": "f64", "n": _log(rng, 1_000, 1_500_000),
                "c": rng.randint(2, 16)}
    if kind == "spmm":
        return {"kind": kind, "store": store, "n": _log(rng, 2_000, 700_000), "c": rng.randint(4, 20),
                "k": rng.choice([2, 4, 7, 8, 12, 16, 24, 32, 33, 48])}
    if kind == "dense":
        return {"kind": kind, "store": store, "rows": _log(rng, 300, 9_000), "cols": _log(rng, 300, 9_000),
                "k": 1 if store == "f64" else rng.choice([1, 1, 8, 33, 64])}
    if kind == "batch":
        return {"kind": kind, "store": store, "count": rng.randint(8, 64), "n_max": _log(rng, 5_000, 100_000)}
    if kind == "pagerank":
        if rng.random() < 0.4:
            return {"kind": kind, "graph": "cqmat", "n": _log(rng, 2_000, 400_000), "c": rng.randint(4, 16),
                    "mode": "reference", "precision": "f64", "accel": 0}
        precision = rng.choice(["f64", "f64", "f32", "bf16"])
        return {"kind": kind, "graph": "rmat", "scale": rng.randint(12, 20), "mode": "dangling",
                "precision": precision, "accel": rng.choice([0, 1])}
    if kind == "ppr":
        precision = rng.choice(["f64", "f32"])
        return {"kind": kind, "scale": rng.randint(12, 16), "k": rng.randint(3, 64), "precision": precision,
                "refined": precision == "f32", "accel": rng.choice([0, 1])}
    if kind == "pagerank_grad":
        return {"kind": kind, "scale": rng.randint(11, 16)}
    return {"kind": kind, "store": rng.choice(["f64", "f32"]), "n": _log(rng, 2_000, 700_000), "c": rng.randint(4, 18)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(count, store, g):
    """Uniform (0, 1], exactly representable in the value store, as FP64."""
    return (1.0 - torch.rand(count, dtype=torch.float32, device="cuda", generator=g)).to(TORCH[store]).double()


def cqmat(n, c, store, g, q=0.1, merge=True):
    """c entries per row on a band starting at the diagonal, each moved to a uniform random
    column with probability q, duplicates merged (or kept, as fill_cqmat leaves them):
    (rowptr, cols, values) on the GPU."""
    c = min(c, n)
    cols = (torch.arange(n, device="cuda")[:, None] + torch.arange(c, device="cuda")[None, :]) % n
    moved = torch.rand((n, c), device="cuda", generator=g) < q
    cols = torch.where(moved, torch.randint(0, n, (n, c), device="cuda", generator=g), cols)
    del moved
    cols = cols.sort(dim=1).values
    keep = torch.ones((n, c), dtype=torch.bool, device="cuda")
    if merge:
        keep[:, 1:] = cols[:, 1:] != cols[:, :-1]
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = keep.sum(dim=1).cumsum(0)
    cols = cols[keep].int()
    return rowptr.int(), cols, _values(cols.numel(), store, g)


def ragged(n, mean, store, g):
    """Log-normal row lengths with 5 % empty rows and one hub row per 20000 of 2000 to 12000
    entries; each entry in a band of 64 columns around the diagonal or anywhere, half each."""
    ln = torch.exp(torch.randn(n, device="cuda", generator=g) * 0.9 + math.log(mean) - 0.405).long()
    ln[torch.rand(n, device="cuda", generator=g) < 0.05] = 0
    hubs = max(1, n // 20_000)
    at = torch.randint(0, n, (hubs,), device="cuda", generator=g)
    ln[at] = torch.randint(2_000, 12_000, (hubs,), device="cuda", generator=g)
    ln.clamp_(max=n)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = ln.cumsum(0)
    nnz = int(rowptr[-1])
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), ln)
    band = (row + torch.randint(-32, 32, (nnz,), device="cuda", generator=g)) % n
    far = torch.randint(0, n, (nnz,), device="cuda", generator=g)
    cols = torch.where(torch.rand(nnz, device="cuda", generator=g) < 0.5, band, far)
    order = (row * n + cols).sort().indices
    return rowptr.int(), cols[order].int(), _values(nnz, store, g)


def rmat(scale, g, merge=True):
    """R-MAT digraph, 16 draws per vertex, (a, b, c, d) = (0.57, 0.19, 0.19, 0.05), repeated
    edges merged (or kept: a multigraph), as the column-stochastic PageRank matrix: row =
    destination, column = source, value 1 / out-degree."""
    n, m = 1 << scale, 16 << scale
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        u = torch.rand(m, device="cuda", generator=g)
        src = src * 2 + (u >= 0.76)
        dst = dst * 2 + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    key = torch.unique(dst * n + src) if merge else (dst * n + src).sort().values
    row, col = key // n, key % n
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.bincount(row, minlength=n).cumsum(0)
    deg = torch.bincount(col, minlength=n)
    return rowptr.int(), col.int(), 1.0 / deg[col].double()


def stochastic(n, c, g):
    """The cqmat pattern with every value 1 divided by its column's sum."""
    rowptr, cols, _ = cqmat(n, c, "f64", g)
    return rowptr, cols, 1.0 / torch.bincount(cols, minlength=n)[cols.long()].double()


def arrays(case, seed):
    """(rows, columns, rowptr, cols, values) of the case's matrix, on the GPU."""
    g = _gen(seed)
    if case["kind"] == "ragged":
        return (case["n"], case["n"], *ragged(case["n"], case["mean"], case["store"], g)), g
    if case["kind"] in ("ppr", "pagerank_grad") or case.get("graph") == "rmat":
        merge = case["kind"] != "pagerank_grad"  # a training program's edges are its own list
        return (1 << case["scale"], 1 << case["scale"], *rmat(case["scale"], g, merge)), g
    if case["kind"] == "pagerank":
        return (case["n"], case["n"], *stochastic(case["n"], case["c"], g)), g
    return (case["n"], case["n"], *cqmat(case["n"], case["c"], case["store"], g, merge=case["kind"] != "spmv_grad")), g


def handle(fmt, n_row, n_col, rowptr, cols, values, stores):
    if fmt == "CSR":
        return capi.DeviceMatrix.csr(n_row, n_col, rowptr.cpu().numpy(), cols.cpu().numpy(), values.cpu().numpy(),
                                     stores=stores)
    length = (rowptr[1:] - rowptr[:-1]).long()
    row = torch.repeat_interleave(torch.arange(n_row, device="cuda"), length)
    if fmt == "COO":
        return capi.DeviceMatrix.coo(n_row, n_col, row.int().cpu().numpy(), cols.cpu().numpy(), values.cpu().numpy(),
                                     stores=stores)
    width = int(length.max())
    slot = torch.arange(cols.numel(), device="cuda") - rowptr[:-1].long()[row]
    ec = torch.zeros((n_row, width), dtype=torch.int32, device="cuda")
    ev = torch.zeros((n_row, width), dtype=torch.float64, device="cuda")
    ec[row, slot] = cols
    ev[row, slot] = values
    return capi.DeviceMatrix.ell(n_row, n_col, width, ec.cpu().numpy().ravel(), ev.cpu().numpy().ravel(),
                                 stores=stores)


def batch_sizes(case):
    rng = np.random.default_rng(case["count"])
    return [(int(np.exp(rng.uniform(np.log(1_000), np.log(case["n_max"])))), int(rng.integers(8, 33)))
            for _ in range(case["count"])]


def seed_sets(case, seed):
    """Seed sets of 1 to 100 random vertices, sizes log-uniform."""
    rng = np.random.default_rng(seed)
    return [rng.integers(0, 1 << case["scale"], int(np.exp(rng.uniform(0, np.log(100))))).astype(np.int32)
            for _ in range(case["k"])]


def vectors(case, n, g):
    """The vectors of a case, drawn after its matrix."""
    kind = case["kind"]
    if kind in ("spmv", "ragged", "axpx_host"):
        return torch.rand(n, dtype=vector_dtype(case["store"]), device="cuda", generator=g)
    if kind == "spmm":
        return torch.rand((n, case["k"]), dtype=vector_dtype(case["store"]), device="cuda", generator=g)
    if kind == "spmv_grad":
        dt = vector_dtype(case["store"])
        return (torch.rand(n, dtype=dt, device="cuda", generator=g),
                torch.randn(n, dtype=dt, device="cuda", generator=g))
    if kind == "pagerank_grad":
        v = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
        return v / v.sum(), torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    return None


def dense_inputs(case, seed):
    g = _gen(seed)
    a = _values(case["rows"] * case["cols"], case["store"], g)
    x = torch.rand((case["k"], case["cols"]), dtype=vector_dtype(case["store"]), device="cuda", generator=g)
    return a.view(case["rows"], case["cols"]), x


def batch_inputs(case, seed):
    g = _gen(seed)
    out = []
    for n, c in batch_sizes(case):
        out.append((n, *cqmat(n, c, case["store"], g),
                    torch.rand(n, dtype=vector_dtype(case["store"]), device="cuda", generator=g)))
    return out


def offsets(sizes):
    """Where each of the vectors begins in their common buffer, and the buffer's size."""
    at, total = [], 0
    for n in sizes:
        at.append(total)
        total += (n + 31) // 32 * 32
    return at, total


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "dense":
        a, x = dense_inputs(case, seed)
        s["A"] = capi.DeviceMatrix.dense(case["rows"], case["cols"], case["rows"], case["cols"],
                                         a.cpu().numpy().ravel(), stores=STORE_BIT[case["store"]])
        s["x"], s["y"] = x, torch.empty((case["k"], case["rows"]), dtype=x.dtype, device="cuda")
        return s
    if kind == "batch":
        inputs = batch_inputs(case, seed)
        # the results stand in one buffer, each member's from a multiple of 32 entries
        at, total = offsets([x.numel() for *_, x in inputs])
        members = [handle("CSR", n, n, rowptr, cols, values, STORE_BIT[case["store"]])
                   for n, rowptr, cols, values, _ in inputs]
        xs = [x for *_, x in inputs]
        y = torch.zeros(total, dtype=xs[0].dtype, device="cuda")
        s["A"], s["x"], s["y"] = capi.Batch(members), xs, y
        s["A"].bind(STORE[case["store"]], [x.data_ptr() for x in xs], [y[a:].data_ptr() for a in at])
        return s
    (n, n_col, rowptr, cols, values), g = arrays(case, seed)
    if kind == "pagerank":
        stores = STORE_BIT["f64"] | STORE_BIT[case["precision"]]
    elif kind == "ppr":
        stores = STORE_BIT["f64"] | (STORE_BIT["f32"] if case["precision"] == "f32" else 0)
    elif kind == "pagerank_grad":
        stores = STORE_BIT["f64"]
    elif kind == "spmv_grad":
        stores = STORE_BIT["f64"] | STORE_BIT[case["store"]]
    else:
        stores = STORE_BIT[case["store"]]
    s["A"] = handle(case.get("fmt", "CSR"), n, n_col, rowptr, cols, values, stores)
    x = vectors(case, n, g)
    if kind in ("spmv", "ragged", "spmm"):
        s["x"], s["y"] = x, torch.empty_like(x)
    elif kind == "axpx_host":
        s["x"] = x.cpu().numpy()
    elif kind == "pagerank":
        s["y"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif kind == "ppr":
        s["sets"] = seed_sets(case, seed)
        s["y"] = torch.empty((case["k"], n), dtype=torch.float64, device="cuda")
    else:
        s["values"] = values.to(x[0].dtype).requires_grad_(True)
        s["x"], s["w"] = x[0].requires_grad_(True), x[1]
    return s


def run(s):
    kind, A = s["kind"], s["A"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind in ("spmv", "ragged") or (kind == "dense" and s["k"] == 1):
        vt = capi.F64 if s["store"] == "f64" else capi.F32
        A.spmv_ex(STORE[s["store"]], vt, s["x"].data_ptr(), vt, s["y"].data_ptr(), 0, stream)
        return s["y"]
    if kind == "axpx_host":
        return A.a_axpx_host(s["x"])
    if kind == "spmm":
        A.spmm(STORE[s["store"]], s["k"], s["x"].data_ptr(), s["k"], s["y"].data_ptr(), s["k"], stream)
        return s["y"]
    if kind == "dense":
        A.dense_spmm(STORE[s["store"]], s["k"], s["x"].data_ptr(), s["cols"], s["y"].data_ptr(), s["rows"], stream)
        return s["y"]
    if kind == "batch":
        A.spmv(stream, graph=True)
        return s["y"]
    if kind == "pagerank":
        if s["mode"] == "reference":
            A.pagerank(s["y"].data_ptr(), beta=0.85, tol=1e-9, max_iter=1000, mode=capi.PR_REFERENCE, stream=stream)
        else:
            A.pagerank(s["y"].data_ptr(), beta=0.85, tol=1e-12, max_iter=2000, mode=capi.PR_DANGLING,
                       precision=STORE[s["precision"]], accel=s["accel"], stream=stream)
        return s["y"]
    if kind == "ppr":
        capi.ppr_batched(A, s["sets"], s["y"].data_ptr(), beta=0.85, tol=1e-12, max_iter=1000,
                         precision=STORE[s["precision"]], refined=s["refined"], accel=s["accel"], stream=stream)
        return s["y"]
    if kind == "pagerank_grad":
        y = autograd.pagerank(A, s["values"], s["x"])
    else:
        y = autograd.csr_spmv(A, s["values"], s["x"])
    gv, gx = torch.autograd.grad(y, (s["values"], s["x"]), s["w"])
    return {"y": y.detach(), "grad_values": gv, "grad_x": gx}


# ------------------------------------------------------------------ floors
def _entries(case):
    """Stored entries of the case's matrix, near enough for a floor."""
    if case["kind"] == "ragged":
        return int(case["n"] * case["mean"] * 0.92) + 7_000 * max(1, case["n"] // 20_000)
    if "scale" in case:
        return int((16 << case["scale"]) * 0.95)
    return case["n"] * case["c"]


def work(case):
    kind = case["kind"]
    if kind == "dense":
        vb = VALUE_BYTES[case["store"]]
        xb = 8 if case["store"] == "f64" else 4
        cells = case["rows"] * case["cols"]
        return {"bytes": cells * vb + (case["rows"] + case["cols"]) * case["k"] * xb, "flops": 2 * cells * case["k"]}
    if kind == "batch":
        vb, xb = VALUE_BYTES[case["store"]], 8 if case["store"] == "f64" else 4
        sizes = batch_sizes(case)
        nnz = sum(n * c for n, c in sizes)
        return {"bytes": nnz * (vb + 4) + sum(n for n, _ in sizes) * (4 + 2 * xb), "flops": 2 * nnz}
    nnz = _entries(case)
    n = 1 << case["scale"] if "scale" in case else case["n"]
    if kind in ("spmv", "ragged", "spmm"):
        vb, xb, k = VALUE_BYTES[case["store"]], 8 if case["store"] == "f64" else 4, case.get("k", 1)
        index = 0 if case.get("fmt") == "ELL" else 4 * n
        return {"bytes": nnz * (vb + 4) + index + 2 * n * k * xb, "flops": 2 * nnz * k}
    if kind == "axpx_host":
        return {"bytes": nnz * 12 + 4 * n + 2 * n * 8, "flops": 4 * nnz + n}
    if kind in ("pagerank", "ppr"):  # the matrix and the result once; at least one sweep
        k = case.get("k", 1)
        return {"bytes": nnz * 12 + 4 * n + n * k * 8, "flops": 2 * nnz * k}
    vb = 8 if kind == "pagerank_grad" else VALUE_BYTES[case["store"]]
    # the pattern, the values and their gradient, x, dL/dy, y, dL/dx
    return {"bytes": nnz * (4 + 2 * vb) + 4 * n + 4 * n * vb, "flops": 6 * nnz}


# ------------------------------------------------------------------ 64 bits
def _sparse(n, n_col, rowptr, cols, values):
    return torch.sparse_csr_tensor(rowptr.long(), cols.long(), values.double(), size=(n, n_col),
                                   check_invariants=False)


def _transpose(n, rowptr, cols, values):
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), (rowptr[1:] - rowptr[:-1]).long())
    order = torch.argsort(cols.long(), stable=True)
    tp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    tp[1:] = torch.bincount(cols.long(), minlength=n).cumsum(0)
    return row, _sparse(n, n, tp, row[order], values[order])


def _times(A, x):
    return (A @ x[:, None])[:, 0] if x.dim() == 1 else A @ x


def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        a, x = dense_inputs(case, seed)
        return x.double() @ a.t()
    if kind == "batch":
        inputs = batch_inputs(case, seed)
        at, total = offsets([x.numel() for *_, x in inputs])
        y = torch.zeros(total, dtype=torch.float64, device="cuda")
        for a, (n, rowptr, cols, values, x) in zip(at, inputs):
            y[a:a + n] = _times(_sparse(n, n, rowptr, cols, values), x.double())
        return y
    (n, n_col, rowptr, cols, values), g = arrays(case, seed)
    A = _sparse(n, n_col, rowptr, cols, values)
    x = vectors(case, n, g)
    if kind in ("spmv", "ragged", "spmm"):
        return _times(A, x.double())
    if kind == "axpx_host":
        return _times(A, _times(A, x) + x).cpu().numpy()
    beta = 0.85
    dangling = (torch.bincount(cols.long(), minlength=n) == 0).double()
    if kind == "pagerank" and case["mode"] == "reference":
        b = torch.ones(n, dtype=torch.float64, device="cuda")
        for _ in range(1000):
            new = beta * _times(A, b) + (1 - beta) / n * b.sum()
            new = new / new.max()
            off = float((new - b).abs().sum())
            b = new
            if off < 1e-9:
                break
        return b / b.sum()
    if kind == "pagerank":
        p = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        for _ in range(220):
            p = beta * _times(A, p) + (beta * (dangling @ p) + (1 - beta) * p.sum()) / n
        return p / p.sum()
    if kind == "ppr":
        sets = seed_sets(case, seed)
        v = torch.zeros((n, case["k"]), dtype=torch.float64, device="cuda")
        for c, nodes in enumerate(sets):
            u = torch.from_numpy(np.unique(nodes)).long().cuda()
            v[u, c] = 1.0 / u.numel()
        p = v.clone()
        for _ in range(220):
            p = beta * _times(A, p) + (beta * (dangling @ p) + (1 - beta)) * v
        return p.t().contiguous()
    x, w = x
    row, T = _transpose(n, rowptr, cols, values)
    if kind == "spmv_grad":
        y = _times(A, x.double())
        return {"y": y, "grad_values": w.double()[row] * x.double()[cols.long()], "grad_x": _times(T, w.double())}
    p = x.clone()
    for _ in range(260):
        p = beta * _times(A, p) + (beta * (dangling @ p) + 1 - beta) * x
    lam = w.clone()
    for _ in range(260):
        lam = beta * _times(T, lam) + beta * dangling * (x @ lam) + w
    return {"y": p, "grad_values": beta * lam[row] * p[cols.long()], "grad_x": (beta * (dangling @ p) + 1 - beta) * lam}

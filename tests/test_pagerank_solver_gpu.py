"""The PageRank solver kernel at the edges of its row classes: rows of every
length at which the class changes (1, 4, 8 or 32 lanes, chunks of eight warps,
rows cut into several chunks), empty rows, CSR and COO items, the ELL layout,
one-block and full grids, and a handle whose values change between solves.

Oracle: the CPU restatement (oracle/tbsla_oracle.c).  One FP64 sweep sums rows
of at most L entries and n-entry masses in another order than the oracle: each
sum is within (length) u of exact, so after s sweeps the vectors, of unit L1
norm, are within s (L + n) u of each other (u = 2^-53); both sides' bounds
added, 2 s (L + n) u.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024,
         1025, 4095, 4096, 4097, 8191, 8192, 8193, 20000]


def graph(rng, n, lens):
    """A column-stochastic n x n matrix with the given row lengths at random
    rows (the others 0 to 6), repeated columns allowed; some columns dangling."""
    ln = rng.integers(0, 7, n)
    ln[rng.permutation(n)[:len(lens)]] = lens
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, max(1, n - n // 8), rp[-1]).astype(np.int32)
    va = 1.0 / np.bincount(ci, minlength=n)[ci]
    return rp, ci, va, (np.bincount(ci, minlength=n) == 0).astype(np.uint8)


@pytest.mark.parametrize("n,lens", [(1, [1]), (40, [4, 9, 33]), (5000, EDGES), (300000, EDGES * 40)])
@pytest.mark.parametrize("fmt", ["CSR", "COO"])
def test_row_classes(gpu, orc, n, lens, fmt):
    rng = np.random.default_rng(n)
    rp, ci, va, dang = graph(rng, n, lens)
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    if fmt == "CSR":
        A = gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=stores)
    else:
        A = gpu.DeviceMatrix.coo(n, n, np.repeat(np.arange(n, dtype=np.int32), np.diff(rp)), ci, va, stores=stores)
    A.tune(gpu.TUNE_PR_RELABEL, 0)
    bound = 2 * 6 * (max(lens) + n) * 2.0 ** -53
    for _ in range(2):  # the second solve finds the workspace of the first
        x, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_DANGLING)
        xo, it, _ = orc.page_rank_dangling(rp, ci, va, dang, 0.85, 0.0, 6)
        assert r.iterations == it == 6
        assert np.abs(x - xo).sum() <= bound, (np.abs(x - xo).sum(), bound)
    o = orc.from_arrays("CSR", n, n, va, rp, ci)
    b, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_REFERENCE)
    bo, _ = o.page_rank(0.0, 0.85, 6)
    assert np.abs(b - bo).sum() <= bound
    xo, _, _ = orc.page_rank_dangling(rp, ci, va, dang, 0.85, 1e-14, 5000)
    xo = xo / math.fsum(xo)
    for prec, accel in ((gpu.F64, 1), (gpu.F32, 0), (gpu.F32, 1), (gpu.BF16, 1)):
        x, r = A.pagerank_host(beta=0.85, tol=1e-11, max_iter=5000, mode=gpu.PR_DANGLING, precision=prec, accel=accel)
        # ||x - G(x)||_1 < tol: within tol / (1 - beta) of the fixed point
        assert r.converged and np.abs(x - xo).sum() <= 1e-11 / 0.15 + bound, (prec, accel)


@pytest.mark.parametrize("fmt", ["ELL", "CSR"])
def test_ell_layout_and_new_values(gpu, orc, fmt):
    """An ELL handle and the ELL-layout copy of a CSR handle (2^16 rows and
    more); then the CSR handle's values are replaced, some by 0 (columns that
    become dangling), and the solve follows."""
    n, c = 70001, 11
    rng = np.random.default_rng(3)
    ci = np.sort(rng.integers(0, n - 9, (n, c)), axis=1).astype(np.int32)
    va = (1.0 / np.bincount(ci.ravel(), minlength=n)[ci]).astype(np.float64)
    rp = (np.arange(n + 1) * c).astype(np.int32)
    A = (gpu.DeviceMatrix.ell(n, n, c, ci, va) if fmt == "ELL"
         else gpu.DeviceMatrix.csr(n, n, rp, ci.ravel(), va.ravel()))
    assert fmt == "ELL" or A.info().slices > 0
    bound = 2 * 6 * (c + n) * 2.0 ** -53

    def check(v):
        used = np.zeros(n, bool)
        used[ci.ravel()[v.ravel() != 0]] = True
        x, _ = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_DANGLING)
        xo, _, _ = orc.page_rank_dangling(rp, ci.ravel(), v.ravel(), (~used).astype(np.uint8), 0.85, 0.0, 6)
        assert np.abs(x - xo).sum() <= bound * max(1.0, np.abs(xo).sum())
    check(va)
    if fmt == "CSR":
        torch = pytest.importorskip("torch")
        va2 = np.where(ci < n // 2, va, 0.0)
        t = torch.from_numpy(va2.ravel()).cuda()
        A.set_values(gpu.F64, t.data_ptr())
        check(va2)


@pytest.mark.parametrize("scale", [1.0, 1e40, 1e-40])
def test_reference_mode_stops_where_the_oracle_does(gpu, orc, scale):
    """The reference mode's normalisation is left to the next sweep, which also
    tests the convergence: every stopping rule (tolerances from one sweep on,
    every small iteration limit) gives the oracle's iteration count, and so do
    maxima far from 1.  With values scaled by 1e40 the teleport term vanishes:
    a sweep then keeps at least 0.8 of the mass (columns without entries), so
    errors grow by less than 0.8^-6 < 4 over six sweeps."""
    n = 3001
    rng = np.random.default_rng(8)
    rp, ci, va, _ = graph(rng, n, [40, 300])
    A, o = gpu.DeviceMatrix.csr(n, n, rp, ci, va * scale), orc.from_arrays("CSR", n, n, va * scale, rp, ci)
    for limit in (1, 2, 3, 4, 6):
        b, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=limit, mode=gpu.PR_REFERENCE)
        bo, it = o.page_rank(0.0, 0.85, limit)
        assert r.iterations == it == limit
        assert np.abs(b - bo).sum() <= 4 * 2 * 6 * (300 + n) * 2.0 ** -53
    if scale == 1e40:
        return
    for tol in (1e4, 300.0, 30.0, 3.0, 0.3, 1e-2, 1e-4, 1e-6):
        b, r = A.pagerank_host(beta=0.85, tol=tol, max_iter=500, mode=gpu.PR_REFERENCE)
        bo, it = o.page_rank(tol, 0.85, 500)
        assert r.iterations == it and r.converged, tol
        assert np.abs(b - bo).sum() <= 2 * it * (300 + n) * 2.0 ** -53


def test_reference_mode_by_products(gpu, orc):
    """2^22 rows of ragged lengths: a product per sweep and a step of the solver,
    against the oracle after six sweeps (the bound of the other tests)."""
    n = 1 << 22
    rng = np.random.default_rng(22)
    rp, ci, va, _ = graph(rng, n, [40])
    A, o = gpu.DeviceMatrix.csr(n, n, rp, ci, va), orc.from_arrays("CSR", n, n, va, rp, ci)
    assert A.info().slices == 0
    for _ in range(2):
        b, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_REFERENCE)
    bo, it = o.page_rank(0.0, 0.85, 6)
    assert r.iterations == it == 6
    assert np.abs(b - bo).sum() <= 4 * 2 * 6 * (40 + n) * 2.0 ** -53


def test_reference_mode_by_products_keeps_no_work_list(gpu):
    """Where the reference mode multiplies by products, the first solve takes its
    vectors (26 bytes a row) and no list of the rows (16 bytes for each that has
    entries, seven eighths here)."""
    torch = pytest.importorskip("torch")
    n = 1 << 22
    rng = np.random.default_rng(22)
    rp, ci, va, _ = graph(rng, n, [40])
    A = gpu.DeviceMatrix.csr(n, n, rp, ci, va)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    A.pagerank(out.data_ptr(), tol=0.0, max_iter=3, mode=gpu.PR_REFERENCE)
    assert free - torch.cuda.mem_get_info()[0] <= 32 * n

"""PageRank sweeps of large graphs of short rows (5 million entries and more), whose rows of
up to 16 or 32 entries take one lane with 16-byte loads: every row length and every
alignment of a row's first entry, neighbouring rows that gather neighbouring entries
and rows that do not, row pointers of CSR and COO, with and without long rows
enough to lower the limit.

Bounds as in test_pagerank_solver_gpu.py: 2 s (L + n) u in L1 after s sweeps, and
tol / (1 - beta) from the fixed point for converged solves.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("long_rows", [False, True])
@pytest.mark.parametrize("mean", [7, 17])
@pytest.mark.parametrize("fmt", ["CSR", "COO"])
def test_short_rows(gpu, orc, fmt, mean, long_rows, near):
    n = 5_400_000 // mean
    rng = np.random.default_rng(mean)
    # lengths 0 to 2 mean, every start modulo 4 and 8 follows
    ln = rng.integers(0, 2 * mean + 1, n)
    ln[:40] = np.arange(40)
    if long_rows:  # a fifth of the entries in rows above 32
        ln[100:100 + 5_400_000 // 5 // 60] = 60
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    rows = np.repeat(np.arange(n, dtype=np.int64), ln)
    ci = ((rows + rng.integers(0, 3 * mean, rp[-1])) % (n - 11) if near else rng.integers(0, n - 11, rp[-1])).astype(np.int32)
    cnt = np.bincount(ci, minlength=n)
    va = 1.0 / cnt[ci]
    assert rp[-1] // (152 * 1024) >= 32  # the classes of a large graph
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    A = (gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=stores) if fmt == "CSR"
         else gpu.DeviceMatrix.coo(n, n, rows.astype(np.int32), ci, va, stores=stores))
    assert A.info().slices == 0
    dang = (cnt == 0).astype(np.uint8)
    bound = 2 * 6 * (max(60, 2 * mean) + n) * 2.0 ** -53
    x, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_DANGLING)
    xo, it, _ = orc.page_rank_dangling(rp, ci, va, dang, 0.85, 0.0, 6)
    assert r.iterations == it and np.abs(x - xo).sum() <= bound
    xo, _, _ = orc.page_rank_dangling(rp, ci, va, dang, 0.85, 1e-13, 400)
    xo = xo / math.fsum(xo)
    for prec, accel in ((gpu.F32, 0), (gpu.F32, 1), (gpu.BF16, 0), (gpu.BF16, 1)):
        x, r = A.pagerank_host(beta=0.85, tol=1e-9, max_iter=5000, mode=gpu.PR_DANGLING, precision=prec, accel=accel)
        assert r.converged and np.abs(x - xo).sum() <= 1e-9 / 0.15 + bound, (prec, accel)


def test_adjoint_on_short_rows(gpu, orc):
    """The transposed copy of a banded matrix of even rows: its rows differ by a few
    entries.  One sweep against numpy in 64 bits: a row of L entries, L + 3 roundings."""
    torch = pytest.importorskip("torch")
    n, c = 400_000, 15
    rng = np.random.default_rng(1)
    ci = (np.arange(n)[:, None] + rng.integers(0, 2 * c, (n, c))) % n
    va = rng.uniform(0, 2.0 / c, (n, c))
    A = gpu.DeviceMatrix.csr(n, n, (np.arange(n + 1) * c).astype(np.int32), ci.ravel().astype(np.int32), va.ravel())
    w = rng.uniform(0, 1, n)
    tw = torch.from_numpy(w).cuda()
    x, gv = torch.full_like(tw, 1.0 / n), torch.empty_like(tw)
    A.pagerank_adjoint(None, x.data_ptr(), tw.data_ptr(), None, gv.data_ptr(), beta=0.85, tol=0.0, max_iter=1)
    used = np.bincount(ci.ravel(), minlength=n) > 0
    lam = 0.85 * np.bincount(ci.ravel(), weights=(va * w[:, None]).ravel(), minlength=n) + w + np.where(
        used, 0.0, 0.85 * w.mean())
    want = (0.85 * (~used).sum() / n + 0.15) * lam
    longest = np.bincount(ci.ravel(), minlength=n).max()
    assert np.all(np.abs(gv.cpu().numpy() - want) <= 4 * (longest + 8) * 2.0 ** -53 * np.abs(want).max())


def test_reference_mode_on_large_banded_graphs(gpu, orc):
    """2^22 rows that gather near each other: walked, not multiplied by products;
    six sweeps and the sweeps to a tolerance against the oracle."""
    n = 1 << 22
    rng = np.random.default_rng(3)
    ln = rng.integers(0, 13, n)
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = ((np.repeat(np.arange(n, dtype=np.int64), ln) + rng.integers(0, 40, rp[-1])) % n).astype(np.int32)
    va = 1.0 / np.bincount(ci, minlength=n)[ci]
    A, o = gpu.DeviceMatrix.csr(n, n, rp, ci, va), orc.from_arrays("CSR", n, n, va, rp, ci)
    b, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=6, mode=gpu.PR_REFERENCE)
    bo, it = o.page_rank(0.0, 0.85, 6)
    assert r.iterations == it == 6
    assert np.abs(b - bo).sum() <= 4 * 2 * 6 * (13 + n) * 2.0 ** -53
    b, r = A.pagerank_host(beta=0.85, tol=100.0, max_iter=200, mode=gpu.PR_REFERENCE)
    bo, it = o.page_rank(100.0, 0.85, 200)
    assert r.iterations == it and r.converged

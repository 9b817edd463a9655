"""PageRank of handles whose products were given another kernel variant (CSR row
blocks, COO merge path, ELL four rows a thread): the solver walks their arrays all
the same, so results and sweep counts are those of the default variant, bit for
bit, in every mode and precision.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 40000])
@pytest.mark.parametrize("fmt", ["CSR", "COO", "SCOO", "ELL"])
def test_variant_makes_no_difference(gpu, fmt, n):
    rng = np.random.default_rng(n)
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    if fmt == "ELL":
        c = 6
        ci = np.sort(rng.integers(0, n, (n, c)), axis=1).astype(np.int32)
        A = gpu.DeviceMatrix.ell(n, n, c, ci, 1.0 / np.bincount(ci.ravel(), minlength=n)[ci], stores=stores)
    else:
        ln = rng.integers(0, 9, n)
        ln[n // 2] = 5 * n if n < 1000 else n // 3
        rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
        ci = rng.integers(0, n, rp[-1]).astype(np.int32)
        va = 1.0 / np.bincount(ci, minlength=n)[ci]
        row = np.repeat(np.arange(n, dtype=np.int32), ln)
        if fmt == "CSR":
            A = gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=stores)
        else:
            A = gpu.DeviceMatrix.coo(n, n, row, ci, va, stores=stores)
            if fmt == "SCOO":
                A = A.to_scoo(stores)
    A.tune(gpu.TUNE_PR_RELABEL, 0)

    def solves():
        kw = [dict(mode=gpu.PR_REFERENCE, tol=1e-9), dict(mode=gpu.PR_DANGLING, tol=1e-12),
              dict(mode=gpu.PR_DANGLING, tol=1e-12, accel=1), dict(mode=gpu.PR_DANGLING, tol=1e-11, precision=gpu.F32),
              dict(mode=gpu.PR_DANGLING, tol=1e-11, precision=gpu.BF16, accel=1)]
        return [(x, r.iterations) for x, r in (A.pagerank_host(max_iter=400, **k) for k in kw)]
    want = solves()
    A.set_variant(1)
    for (x, it), (xw, itw) in zip(solves(), want):
        assert it == itw and np.array_equal(x, xw)

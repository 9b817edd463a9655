"""Reference mode on matrices whose every iterate is negative before its
normalisation: dividing by a negative maximum turns the vector round, and the
solve stops where the oracle's does.

Matrix: minus a dense positive column-stochastic one; a sweep maps 1 to -0.85 +
0.15, so relative errors grow by at most 1 / 0.7 a sweep, and each sweep adds
(L + n) u (L = n entries a row, u = 2^-53).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["CSR", "COO", "ELL", "DENSE"])
@pytest.mark.parametrize("n", [50, 300])
def test_negative_maxima(gpu, orc, n, fmt):
    rng = np.random.default_rng(n)
    a = rng.uniform(0.2, 1, (n, n))
    a = -a / a.sum(0)
    rp, ci = (np.arange(n + 1) * n).astype(np.int32), np.tile(np.arange(n, dtype=np.int32), n)
    o = orc.from_arrays("CSR", n, n, a.ravel(), rp, ci)
    if fmt == "CSR":
        A = gpu.DeviceMatrix.csr(n, n, rp, ci, a.ravel())
    elif fmt == "COO":
        A = gpu.DeviceMatrix.coo(n, n, np.repeat(np.arange(n, dtype=np.int32), n), ci, a.ravel())
    elif fmt == "ELL":
        A = gpu.DeviceMatrix.ell(n, n, n, ci, a.ravel())
    else:
        A = gpu.DeviceMatrix.dense(n, n, n, n, a.ravel())
    for tol, limit in ((0.0, 1), (0.0, 2), (0.0, 3), (0.0, 8), (0.1, 200), (1e-3, 200), (1e-6, 200), (1e-9, 200)):
        b, r = A.pagerank_host(beta=0.85, tol=tol, max_iter=limit, mode=gpu.PR_REFERENCE)
        bo, it = o.page_rank(tol, 0.85, limit)
        assert (r.iterations, r.converged) == (it, int(tol > 0)), (tol, limit)
        assert np.abs(b - bo).sum() <= 2 * it * (n + n) * 2.0 ** -53 * 0.7 ** -it

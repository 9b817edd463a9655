"""The grid barriers of the PageRank solver: a long wait is not a lost one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_sweep_of_seconds_is_waited_for(gpu):
    """Four rows of 20 million slots: four lanes walk them for seconds while
    every other block of the grid waits at the barrier.  The matrix is column
    stochastic and its sweep maps 1/n to 1/n; a sum of w rounded terms is within w
    u of exact (relative), u = 2^-53."""
    n, w = 4, 20_000_000
    cols = np.broadcast_to(np.arange(w, dtype=np.int32) % n, (n, w))
    A = gpu.DeviceMatrix.ell(n, n, w, cols, np.full((n, w), 1.0 / w))
    x, r = A.pagerank_host(beta=0.85, tol=0.0, max_iter=1, mode=gpu.PR_DANGLING)
    assert r.iterations == 1
    assert np.abs(x - 1.0 / n).max() <= 2 * w * 2.0 ** -53 / n

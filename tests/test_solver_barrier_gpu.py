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


def test_handle_is_usable_after_a_lost_barrier(gpu, orc):
    """With few polls a wait runs out at once or in any later sweep, while other
    blocks go on: the solve ends with TBSLA_ERR_TIMEOUT (or, where no wait was
    that long, with its result).  The next solve on the handle is right, and has
    the bits of one on a new handle: rows of several chunks (their arrival counts
    are kept between launches), the adjoint on the transposed copy, the
    mixed-precision solve with its queued launches."""
    torch = pytest.importorskip("torch")
    n = 60000
    rng = np.random.default_rng(4)
    ln = rng.integers(0, 9, n)
    ln[rng.permutation(n)[:12]] = 60000
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, n - 50, rp[-1]).astype(np.int32)
    ci[:: 7] = 5  # a long row of the transposed matrix
    cnt = np.bincount(ci, minlength=n)
    va = 1.0 / cnt[ci]
    w = torch.from_numpy(rng.uniform(-1, 1, n)).cuda()
    xs = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    out = torch.empty(n, dtype=torch.float64, device="cuda")

    def solves(M):
        def adjoint():
            M.pagerank_adjoint(None, xs.data_ptr(), w.data_ptr(), None, out.data_ptr(), tol=0.0, max_iter=9)
            return out.cpu().numpy()
        return [lambda: M.pagerank_host(tol=0.0, max_iter=9, mode=gpu.PR_DANGLING)[0],
                lambda: M.pagerank_host(tol=0.0, max_iter=9, mode=gpu.PR_REFERENCE)[0],
                lambda: M.pagerank_host(tol=1e-10, mode=gpu.PR_DANGLING, precision=gpu.F32)[0],
                lambda: M.pagerank_host(tol=0.0, max_iter=9, mode=gpu.PR_DANGLING, accel=1)[0], adjoint]
    stores = gpu.STORE_F64 | gpu.STORE_F32
    A, B = (gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=stores) for _ in range(2))
    want = [f() for f in solves(B)]
    xo, _, _ = orc.page_rank_dangling(rp, ci, va, (cnt == 0).astype(np.uint8), 0.85, 0.0, 9)
    assert np.abs(want[0] - xo).sum() <= 2 * 9 * (60000 + n) * 2.0 ** -53
    lost = [0] * len(want)
    for polls in (1, 2, 5, 12, 30, 70, 150, 400):
        for i, f in enumerate(solves(A)):
            A.tune(gpu.TUNE_SOLVER_POLLS, polls)
            try:
                assert np.array_equal(f(), want[i])
            except gpu.TbslaError as e:
                assert e.status == 5  # TBSLA_ERR_TIMEOUT
                lost[i] += 1
            A.tune(gpu.TUNE_SOLVER_POLLS, 0)
            assert np.array_equal(f(), want[i]), (polls, i)
    assert all(lost), lost  # one poll is less than any wait of this grid

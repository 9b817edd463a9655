"""Copies that a handle builds on first use, with little device memory left: what
fits beside the handle can also be built."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Ballast:
    """Holds the free device memory but `leave` bytes while the block runs."""

    def __init__(self, leave):
        self.leave, self.held = leave, []

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        step = 1 << 34
        while step >= 1 << 21:
            free = torch.cuda.mem_get_info()[0] - self.leave
            if free < step:
                step //= 2
                continue
            self.held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        return self

    def __exit__(self, *exc):
        self.held.clear()
        torch.cuda.empty_cache()


def ragged(rng, n, nnz):
    """rows of uneven lengths (no ELL-layout copy), long ones among them"""
    ln = rng.multinomial(nnz - 3000, np.repeat([0.5, 1.5], [n // 2, n - n // 2]) / n)
    ln[7] += 3000
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    return rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1])


def test_transposed_copy_where_its_entries_fit(gpu):
    """The copy and its map take 16 bytes an entry (FP64); 24 are left."""
    n, nnz = 1 << 18, 1 << 24
    rng = np.random.default_rng(2)
    rp, ci, va = ragged(rng, n, nnz)
    A, B = (gpu.DeviceMatrix.csr(n, n, rp, ci, va) for _ in range(2))
    x = torch.from_numpy(rng.uniform(-1, 1, n)).cuda()
    want, y = torch.empty_like(x), torch.empty_like(x)
    B.spmv_transpose_ex(gpu.F64, gpu.F64, x.data_ptr(), gpu.F64, want.data_ptr())
    torch.cuda.synchronize()
    B.close()
    with Ballast(24 * nnz + (64 << 20)):
        A.spmv_transpose_ex(gpu.F64, gpu.F64, x.data_ptr(), gpu.F64, y.data_ptr())
        torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_relabelled_copy_where_its_entries_fit(gpu):
    """The copy takes 12 bytes an entry and 40 a row, its solve as much a row
    again; 24 an entry are left."""
    scale, nnz = 18, 1 << 24
    n = 1 << scale
    A, B = (gpu.DeviceMatrix.rmat_pagerank(scale, nnz) for _ in range(2))
    for M in (A, B):
        M.tune(gpu.TUNE_PR_RELABEL, 1)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    want = torch.empty_like(out)
    B.pagerank(want.data_ptr(), tol=0.0, max_iter=5, mode=gpu.PR_DANGLING)
    B.close()
    with Ballast(24 * A.info().stored + (64 << 20)):
        A.pagerank(out.data_ptr(), tol=0.0, max_iter=5, mode=gpu.PR_DANGLING)
    assert torch.equal(out, want)


@pytest.mark.parametrize("scale,relabel", [(20, -1), (18, 1)])
def test_solves_without_room_for_the_relabelled_copy(gpu, scale, relabel):
    """The copy only makes a solve faster: with less memory than its build needs
    (10 bytes an entry are left, it sorts 16) the handle itself is swept.  Both
    orders of summation are within s (L + n) u of exact after s sweeps (L entries
    in the longest row, u = 2^-53)."""
    from tbsla_gb300 import capi
    n, nnz, sweeps = 1 << scale, 1 << 24, 5
    A = gpu.DeviceMatrix.rmat_pagerank(scale, nnz)
    longest = int(np.diff(A.csr_download()[0]).max())
    out, want, ppr = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(3))
    A.tune(gpu.TUNE_PR_RELABEL, 0)
    A.pagerank(want.data_ptr(), tol=0.0, max_iter=sweeps, mode=gpu.PR_DANGLING)
    capi.ppr_batched(A, [[5]], ppr.data_ptr(), tol=0.0, max_iter=sweeps)
    want_ppr, bound = ppr.clone(), 2 * sweeps * (longest + n) * 2.0 ** -53
    A.tune(gpu.TUNE_PR_RELABEL, relabel)
    for _ in range(2):
        with Ballast(10 * A.info().stored):
            A.pagerank(out.data_ptr(), tol=0.0, max_iter=sweeps, mode=gpu.PR_DANGLING)
            capi.ppr_batched(A, [[5]], ppr.data_ptr(), tol=0.0, max_iter=sweeps)
            torch.cuda.synchronize()
        assert float((out - want).abs().sum()) <= bound and float((ppr - want_ppr).abs().sum()) <= bound

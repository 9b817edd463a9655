"""The PageRank solves run on a stream of their own: what the caller queued on
its stream comes first, on the legacy stream (NULL) too.  A long kernel holds the
inputs back; the solve on a handle whose buffers all exist must wait for it and
give, bit for bit, what it gives for inputs that are in place.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HOLD = 200_000_000  # clock cycles, about a tenth of a second


@pytest.fixture(scope="module")
def handle(gpu):
    n = 4000
    rng = np.random.default_rng(1)
    ln = rng.integers(0, 12, n)
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    va = 1.0 / np.bincount(ci, minlength=n)[ci]
    return gpu.DeviceMatrix.csr(n, n, rp, ci, va), n, int(rp[-1]), rng


def streams():
    own = torch.cuda.Stream()
    return [(None, torch.cuda.default_stream()), (0, torch.cuda.default_stream()), (own.cuda_stream, own)]


@pytest.mark.parametrize("which", [0, 1, 2])
def test_teleport_waits_for_its_vector(gpu, handle, which):
    A, n, _, rng = handle
    arg, stream = streams()[which]
    v = torch.from_numpy(rng.dirichlet(np.ones(n))).cuda()
    late, want, x = torch.full_like(v, 1.0 / n), torch.empty_like(v), torch.empty_like(v)
    A.pagerank_teleport(v.data_ptr(), want.data_ptr(), tol=1e-13)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(HOLD)
        late.copy_(v)
        A.pagerank_teleport(late.data_ptr(), x.data_ptr(), tol=1e-13, stream=arg)
    torch.cuda.synchronize()
    assert torch.equal(x, want)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_adjoint_waits_for_its_gradient(gpu, handle, which):
    A, n, nnz, rng = handle
    arg, stream = streams()[which]
    x, w = (torch.from_numpy(rng.uniform(-1, 1, n)).cuda() for _ in range(2))
    late = torch.zeros_like(w)
    out = [(torch.empty(nnz, dtype=torch.float64, device="cuda"), torch.empty_like(x)) for _ in range(2)]

    def solve(rhs, o, st):
        A.pagerank_adjoint(None, x.data_ptr(), rhs.data_ptr(), o[0].data_ptr(), o[1].data_ptr(), tol=1e-9, stream=st)
    solve(w, out[0], None)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(HOLD)
        late.copy_(w)
        solve(late, out[1], arg)
    torch.cuda.synchronize()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("which", [0, 1, 2])
def test_result_waits_for_its_readers(gpu, handle, which):
    A, n, _, _ = handle
    arg, stream = streams()[which]
    x, seen = torch.full((n,), 7.0, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    A.pagerank_host(mode=gpu.PR_DANGLING)  # the solve's buffers
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(HOLD)
        seen.copy_(x)
        A.pagerank(x.data_ptr(), mode=gpu.PR_DANGLING, stream=arg)
    torch.cuda.synchronize()
    assert bool((seen == 7.0).all()) and not bool((x == 7.0).any())

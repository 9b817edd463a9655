"""What a handle builds on first use, asked for by several threads at once, is
built once: every thread gets the products and solves of a handle used by one
thread alone, bit for bit, and the handle holds the same device memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

THREADS = 8


def at_once(f):
    gate, errors = threading.Barrier(THREADS), []

    def go(i):
        try:
            gate.wait()
            f(i)
        except Exception as e:  # raised in the test's own thread below
            errors.append(e)
    ts = [threading.Thread(target=go, args=(i,)) for i in range(THREADS)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()


@pytest.mark.parametrize("relabel", [0, 1])
def test_batched_solves(gpu, relabel):
    from tbsla_gb300 import capi
    n, seeds = 1 << 12, [[3], [100, 7], [4000]]
    outs = [torch.empty(len(seeds) * n, dtype=torch.float64, device="cuda") for _ in range(THREADS)]
    streams = [torch.cuda.Stream().cuda_stream for _ in range(THREADS)]
    for _ in range(6):
        A, B = (gpu.DeviceMatrix.rmat_pagerank(12, 16 * n) for _ in range(2))
        for M in (A, B):
            M.tune(gpu.TUNE_PR_RELABEL, relabel)
        want = torch.empty_like(outs[0])
        capi.ppr_batched(B, seeds, want.data_ptr(), tol=1e-10)
        at_once(lambda i: capi.ppr_batched(A, seeds, outs[i].data_ptr(), tol=1e-10, stream=streams[i]))
        assert all(torch.equal(o, want) for o in outs)
        assert A.info().device_bytes == B.info().device_bytes


def test_transposed_products(gpu):
    n = 5000
    rng = np.random.default_rng(6)
    ln = rng.integers(0, 60, n)
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci, va = rng.integers(0, n, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1])
    x = torch.from_numpy(rng.uniform(-1, 1, n)).cuda()
    outs = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(THREADS)]
    streams = [torch.cuda.Stream().cuda_stream for _ in range(THREADS)]
    torch.cuda.synchronize()
    free = []
    for _ in range(6):
        A = gpu.DeviceMatrix.csr(n, n, rp, ci, va)
        at_once(lambda i: A.spmv_transpose_ex(gpu.F64, gpu.F64, x.data_ptr(), gpu.F64, outs[i].data_ptr(), streams[i]))
        want = outs[0].clone()
        assert all(torch.equal(o, want) for o in outs)
        A.close()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[-1] >= free[1], free  # nothing is left behind

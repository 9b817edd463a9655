"""Matrices with long rows: the one-launch product (every row class and the
short rows together) and the values gradient by entry segments, at the row
lengths where a class or a segment changes.

Products against numpy in FP64: a row of L entries is within (L + 1) u of
exact relative to sum |a x| (u = 2^-53 for FP64, 2^-24 for the FP32 sums of
the F32 / BF16 stores, whose values are exact here).  The gradient is one
product per entry: bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES = [0, 1, 2, 7, 8, 9, 31, 32, 33, 95, 96, 97, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025, 8191, 8192, 8193,
         16385, 30000]


def matrix(n, lens, seed):
    rng = np.random.default_rng(seed)
    ln = rng.integers(0, 33, n)
    ln[: len(lens)] = lens
    ln = ln[rng.permutation(n)]
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    va = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    va = torch.from_numpy(va).bfloat16().double().numpy()  # exact in every store
    return rp, ci, va, rng


@pytest.mark.parametrize("n,lens,mode", [(1, [40], -1), (70, EDGES, -1), (5000, EDGES, 0), (5000, EDGES, 2),
                                         (200003, EDGES * 5, -1), (30, [33] * 30, -1)])
@pytest.mark.parametrize("fmt", ["CSR", "COO"])
def test_product_of_mixed_rows(gpu, n, lens, mode, fmt):
    lens = lens[:n]
    rp, ci, va, rng = matrix(n, lens, n + len(lens))
    row = np.repeat(np.arange(n), np.diff(rp)).astype(np.int32)
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    A = (gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=stores) if fmt == "CSR"
         else gpu.DeviceMatrix.coo(n, n, row, ci, va, stores=stores))
    A.tune(gpu.TUNE_SHORT_ROWS, mode)
    assert A.info().kernels == 1 + int(np.diff(rp).max() > 8192)
    x = rng.uniform(-1, 1, n).astype(np.float32).astype(np.float64)
    terms = va * x[ci]
    exact = np.bincount(row, terms, n)
    mass = np.bincount(row, np.abs(terms), n)
    for store, vt, tdt, u in ((gpu.F64, gpu.F64, torch.float64, 2.0 ** -53), (gpu.F32, gpu.F32, torch.float32, 2.0 ** -24),
                              (gpu.BF16, gpu.F32, torch.float32, 2.0 ** -24)):
        tx = torch.from_numpy(x).cuda().to(tdt)
        ty = torch.full((n,), 7.0, dtype=tdt, device="cuda")
        A.spmv_ex(store, vt, tx.data_ptr(), vt, ty.data_ptr())
        y = ty.double().cpu().numpy()
        # numpy's own sum is within (L + 1) 2^-53
        bound = (np.diff(rp) + 2) * (u + 2.0 ** -53) * mass
        assert (np.abs(y - exact) <= bound).all(), (store, np.max(np.abs(y - exact) - bound))
    if fmt == "CSR":
        a, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        for tdt, code in ((np.float64, gpu.F64), (np.float32, gpu.F32)):
            ta, tb = torch.from_numpy(a.astype(tdt)).cuda(), torch.from_numpy(b.astype(tdt)).cuda()
            out = torch.full((max(ci.size, 1),), 7.0, dtype=ta.dtype, device="cuda")
            A.grad_values(code, ta.data_ptr(), tb.data_ptr(), 0.75, out.data_ptr())
            want = (tdt(0.75) * a.astype(tdt))[row] * b.astype(tdt)[ci]
            assert np.array_equal(out.cpu().numpy()[: ci.size], want)

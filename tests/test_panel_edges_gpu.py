"""DENSE products and k-vector products at the sizes where their kernels take
another path: column counts with and without 16-byte rows, few and many rows
(the columns of a row group split over warps), unaligned vectors; panel widths
with and without 16-byte vectors, rows that begin at every offset from a
multiple of four entries, leading dimensions that forbid 16-byte stores.

Against numpy in FP64 on inputs exact in every store: a sum of L products is
within (L + 1) u of exact relative to sum |a x| (u = 2^-53, FP32 2^-24).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = (("F64", torch.float64, 2.0 ** -53), ("F32", torch.float32, 2.0 ** -24), ("BF16", torch.float32, 2.0 ** -24))


def exact_values(rng, shape):
    """Uniform values that BF16 holds exactly."""
    v = torch.from_numpy(rng.uniform(-1, 1, shape).astype(np.float32))
    return v.bfloat16().double().numpy()


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (2, 8192), (17, 8200), (300, 1031), (301, 1032), (5000, 127),
                                       (5001, 128), (9000, 6), (40, 20000), (2433, 1024)])
@pytest.mark.parametrize("shift", [0, 1])
def test_dense_product_edges(gpu, rows, cols, shift):
    rng = np.random.default_rng(rows * 7 + cols)
    a = exact_values(rng, (rows, cols))
    x = exact_values(rng, cols)
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    A = gpu.DeviceMatrix.dense(rows, cols, rows, cols, a.ravel(), stores=stores)
    exact, mass = a @ x, np.abs(a) @ np.abs(x)
    for name, tdt, u in CASES:
        vt = gpu.F64 if name == "F64" else gpu.F32
        buf = torch.empty(cols + 1, dtype=tdt, device="cuda")
        tx = buf[shift:shift + cols]  # shift 1: x off its 16-byte boundary
        tx.copy_(torch.from_numpy(x))
        y = torch.full((rows,), 7.0, dtype=tdt, device="cuda")
        A.spmv_ex(getattr(gpu, name), vt, tx.data_ptr(), vt, y.data_ptr())
        off = np.abs(y.double().cpu().numpy() - exact)
        assert (off <= (cols + 2) * (u + 2.0 ** -53) * mass).all(), (name, off.max())


@pytest.mark.parametrize("k,pad", [(1, 0), (2, 0), (3, 1), (4, 0), (7, 0), (8, 3), (16, 0), (16, 1), (20, 4), (31, 0),
                                   (32, 0), (33, 0), (64, 4)])
def test_panel_edges(gpu, k, pad):
    rng = np.random.default_rng(k * 10 + pad)
    n = 2003
    ln = rng.integers(0, 12, n)
    ln[5], ln[77] = 700, 33
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    assert set(rp[:-1] % 4) == {0, 1, 2, 3}
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    va = exact_values(rng, rp[-1])
    row = np.repeat(np.arange(n), ln)
    A = gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16)
    x = exact_values(rng, (n, k))
    exact, mass = np.zeros((n, k)), np.zeros((n, k))
    np.add.at(exact, row, va[:, None] * x[ci])
    np.add.at(mass, row, np.abs(va[:, None] * x[ci]))
    for name, tdt, u in CASES:
        X = torch.zeros((n, k + pad), dtype=tdt, device="cuda")
        X[:, :k] = torch.from_numpy(x)
        Y = torch.full((n, k + pad), 7.0, dtype=tdt, device="cuda")
        A.spmm(getattr(gpu, name), k, X.data_ptr(), k + pad, Y.data_ptr(), k + pad)
        y = Y.double().cpu().numpy()
        assert (y[:, k:] == 7.0).all()
        assert (np.abs(y[:, :k] - exact) <= (ln[:, None] + 2) * (u + 2.0 ** -53) * mass).all(), name

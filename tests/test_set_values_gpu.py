"""tbsla_matrix_set_values: every store of the handle, its ELL-layout copy and
its transposed copy follow new FP64 or FP32 values.  Products of the updated
handle equal those of a handle created with the values, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rows(kind, rng):
    if kind == "even":      # keeps the ELL-layout copy (2^16 rows and more)
        return np.full(65536 + 37, 9)
    if kind == "longest":   # rows of 32 entries: the largest tiles
        return np.full(65536 + 1, 32)
    if kind == "short":     # no copy
        return rng.integers(0, 33, 1000)
    ln = rng.integers(0, 40, 3001)  # long rows too
    ln[7], ln[2999] = 9000, 300
    return ln


@pytest.mark.parametrize("kind", ["even", "longest", "short", "mixed"])
@pytest.mark.parametrize("dtype", ["F64", "F32"])
def test_new_values_reach_every_copy(gpu, kind, dtype):
    rng = np.random.default_rng(11)
    ln = rows(kind, rng)
    n = ln.size
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    stores = gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16
    new = rng.uniform(-1, 1, rp[-1]).astype(np.float64 if dtype == "F64" else np.float32)
    A = gpu.DeviceMatrix.csr(n, n, rp, ci, rng.uniform(-1, 1, rp[-1]), stores=stores)
    B = gpu.DeviceMatrix.csr(n, n, rp, ci, new.astype(np.float64), stores=stores)
    assert (A.info().slices > 0) == (kind in ("even", "longest"))

    def products(M):
        out = []
        for store, vt, tdt in ((gpu.F64, gpu.F64, torch.float64), (gpu.F32, gpu.F32, torch.float32),
                               (gpu.BF16, gpu.F32, torch.float32)):
            x = torch.from_numpy(x0).cuda().to(tdt)
            for f in (M.spmv_ex, M.spmv_transpose_ex):
                y = torch.empty(n, dtype=tdt, device="cuda")
                f(store, vt, x.data_ptr(), vt, y.data_ptr())
                out.append(y.cpu().numpy())
        return out
    x0 = rng.uniform(-1, 1, n)
    products(A)  # builds the transposed copy with the old values
    t = torch.from_numpy(new).cuda()
    A.set_values(gpu.F64 if dtype == "F64" else gpu.F32, t.data_ptr())
    for a, b in zip(products(A), products(B)):
        assert np.array_equal(a, b)

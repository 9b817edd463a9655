"""Products of matrices with thousands of rows between 1024 and 1792 entries: one
row fewer than fills the GPU with warps, exactly as many, and one more, with
rows on both sides of either limit, against scipy.

Bound: a sum of L products, each rounded once and added in any order, is within
(L + 1) u sum|a x| of exact (u = 2^-53 or 2^-24 of the stored values; both sides)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
sp = pytest.importorskip("scipy.sparse")


@pytest.mark.parametrize("many", [8191, 8192, 8193])
def test_rows_by_warp_or_block(gpu, many):
    rng = np.random.default_rng(many)
    ln = np.concatenate([np.where(np.arange(many) % 2, 1025, 1026), [0, 1, 32, 33, 1023, 1024, 1793, 2049, 4000, 9000]])
    ln[5] = 1792
    assert int(((ln > 1024) & (ln <= 1792)).sum()) == many
    rng.shuffle(ln)
    n, m = ln.size, 4096
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci, va = rng.integers(0, m, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1])
    x = rng.uniform(-1, 1, m)
    A = gpu.DeviceMatrix.csr(n, m, rp, ci, va, stores=gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16)
    for store, vt, dt, u in ((gpu.F64, gpu.F64, np.float64, 2.0 ** -53), (gpu.F32, gpu.F32, np.float32, 2.0 ** -24),
                             (gpu.BF16, gpu.F32, np.float32, 2.0 ** -24)):
        v = va.astype(dt)
        if store == gpu.BF16:
            v = torch.from_numpy(va).to(torch.bfloat16).double().numpy()
        xs = x.astype(dt)
        v, x64 = v.astype(np.float64), xs.astype(np.float64)
        want = sp.csr_matrix((v, ci, rp), shape=(n, m)) @ x64
        scale = sp.csr_matrix((np.abs(v), ci, rp), shape=(n, m)) @ np.abs(x64)
        tx = torch.from_numpy(xs).cuda()
        y = torch.empty(n, dtype=tx.dtype, device="cuda")
        A.spmv_ex(store, vt, tx.data_ptr(), vt, y.data_ptr())
        err = np.abs(y.cpu().numpy().astype(np.float64) - want)
        assert np.all(err <= 2 * (ln + 2) * u * scale)

"""The ELL-layout copies that batches read smaller members from belong to the
batches: none where the handle's copy was dropped, none for a store that does not read
them, shared, freed with the last batch, and current after new values.  Every
product equals the CSR arrays' thread-per-row product (TBSLA_TUNE_SHORT_ROWS 0)
bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def even(gpu, n, c, rng):
    ci = np.sort(rng.integers(0, n, (n, c)), axis=1).astype(np.int32)
    rp = (np.arange(n + 1) * c).astype(np.int32)
    return gpu.DeviceMatrix.csr(n, n, rp, ci.ravel(), rng.uniform(-1, 1, n * c),
                                stores=gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16)


STORES = [("F64", "F64", torch.float64), ("F32", "F32", torch.float32), ("BF16", "F32", torch.float32)]


def products(gpu, B, Ms, store, bind=True):
    s, vt, dt = next((getattr(gpu, a), getattr(gpu, b), t) for a, b, t in STORES if a == store)
    xs = [torch.linspace(-1, 1, M.info().n_col, dtype=dt, device="cuda") for M in Ms]
    ys = [torch.full_like(x, 9.0) for x in xs]
    want = [torch.full_like(x, 9.0) for x in xs]
    if bind:
        B.bind(s, [x.data_ptr() for x in xs], [y.data_ptr() for y in ys])
        B.kept = (xs, ys)
    xs, ys = B.kept
    B.spmv()
    for M, x, w in zip(Ms, xs, want):
        M.tune(gpu.TUNE_SHORT_ROWS, 0)
        M.spmv_ex(s, vt, x.data_ptr(), vt, w.data_ptr())
        M.tune(gpu.TUNE_SHORT_ROWS, -1)
    torch.cuda.synchronize()
    assert all(torch.equal(y, w) for y, w in zip(ys, want)), store


def held(Ms):
    return [M.info().device_bytes for M in Ms]


@pytest.mark.parametrize("n", [300, 65535, 65536])
def test_dropped_copies_stay_dropped(gpu, n):
    rng = np.random.default_rng(n)
    Ms = [even(gpu, n, 7, rng) for _ in range(2)]
    for M in Ms:
        M.tune(gpu.TUNE_DROP_SLICED_COPY, 1)
    before = held(Ms)
    B = gpu.Batch(Ms)
    for store in ("F64", "F32", "BF16"):
        products(gpu, B, Ms, store)
        assert held(Ms) == before
    B.close()


def test_copies_live_and_die_with_their_batches(gpu):
    rng = np.random.default_rng(5)
    Ms = [even(gpu, n, c, rng) for n, c in ((256, 4), (257, 32), (3000, 9), (60001, 5))]
    before = held(Ms)
    B = gpu.Batch(Ms)
    slots = [(n + 31) // 32 * 32 * c for n, c in ((256, 4), (257, 32), (3000, 9), (60001, 5))]
    # the columns, where rounding the rows up to 32 adds at most 1/32 (257 rows: none)
    assert [b - a for a, b in zip(before, held(Ms))] == [64 + 4 * s if i != 1 else 0 for i, s in enumerate(slots)]
    products(gpu, B, Ms, "BF16")
    assert held(Ms) == before                       # BF16 reads the CSR arrays
    products(gpu, B, Ms, "F32")
    one = held(Ms)
    # and the FP32 values
    assert [b - a for a, b in zip(before, one)] == [2 * 64 + 8 * s if i != 1 else 0 for i, s in enumerate(slots)]
    C = gpu.Batch(Ms[1:])
    products(gpu, C, Ms[1:], "F32")
    assert held(Ms) == one                          # shared
    products(gpu, C, Ms[1:], "F64")
    assert held(Ms)[0] == one[0] and held(Ms)[2] > one[2]
    new = [torch.rand(M.info().stored, dtype=torch.float64, device="cuda") for M in Ms]
    torch.cuda.synchronize()
    for M, v in zip(Ms, new):
        M.set_values(gpu.F64, v.data_ptr())
    products(gpu, B, Ms, "F32", bind=False)          # the bound copies follow new values
    products(gpu, C, Ms[1:], "F64", bind=False)
    Ms[2].tune(gpu.TUNE_DROP_SLICED_COPY, 1)
    products(gpu, B, Ms, "F32", bind=False)          # a bound batch keeps its copy
    B.close()
    C.close()
    assert held(Ms) == before
    B = gpu.Batch(Ms)
    products(gpu, B, Ms, "F64")
    assert held(Ms)[2] == before[2] and held(Ms)[3] > before[3]
    for M in Ms:                                     # members may go first
        M.close()
    B.close()

"""The copies a handle builds on the device on first use: the transposed copy
of blocks (column offset, rows the block does not store, empty rows and
columns, repeated columns, no entries at all) and the degree-relabelled copy
of small forced cases.  The transposed product adds a column's entries in row
order: with integer values the sums are exact."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_row,n_col,f_col,rows,nnz", [(1, 1, 0, 1, 1), (5, 9, 0, 5, 0), (40, 30, 100, 33, 200),
                                                        (3000, 5, 7, 3000, 20000), (7, 70001, 0, 7, 40000),
                                                        (1025, 1024, 1, 1024, 5000)])
def test_transposed_copy_of_blocks(gpu, n_row, n_col, f_col, rows, nnz):
    rng = np.random.default_rng(nnz + n_col)
    row = np.sort(rng.integers(0, rows, nnz))
    rp = np.searchsorted(row, np.arange(rows + 1)).astype(np.int32)
    ci = rng.integers(0, n_col, nnz).astype(np.int32)
    va = rng.integers(-9, 10, nnz).astype(np.float64)
    A = gpu.DeviceMatrix.csr(n_row, n_col, rp, ci + f_col, va, f_col=f_col, stores=gpu.STORE_F64 | gpu.STORE_F32,
                             rows=rows)
    x = rng.integers(-9, 10, n_row).astype(np.float64)
    want = np.bincount(ci, va * x[row], n_col) if nnz else np.zeros(n_col)
    for store, vt, tdt in ((gpu.F64, gpu.F64, torch.float64), (gpu.F32, gpu.F32, torch.float32)):
        tx = torch.from_numpy(x).cuda().to(tdt)
        y = torch.full((n_col,), 5.0, dtype=tdt, device="cuda")
        for _ in range(2):
            A.spmv_transpose_ex(store, vt, tx.data_ptr(), vt, y.data_ptr())
            assert np.array_equal(y.double().cpu().numpy(), want)


@pytest.mark.parametrize("n,nnz", [(1, 1), (2, 5), (1000, 40000), (4097, 9000)])
def test_relabelled_copy(gpu, orc, n, nnz):
    rng = np.random.default_rng(n)
    row = np.sort((n * rng.random(nnz) ** 3).astype(np.int64))
    rp = np.searchsorted(row, np.arange(n + 1)).astype(np.int32)
    ci = (n * rng.random(nnz) ** 2).astype(np.int32)  # repeated columns among them
    va = 1.0 / np.bincount(ci, minlength=n)[ci]
    dang = (np.bincount(ci, minlength=n) == 0).astype(np.uint8)
    A = gpu.DeviceMatrix.csr(n, n, rp, ci, va, stores=gpu.STORE_F64 | gpu.STORE_F32)
    A.tune(gpu.TUNE_PR_RELABEL, 1)
    xo, _, _ = orc.page_rank_dangling(rp, ci, va, dang, 0.85, 1e-14, 5000)
    xo = xo / math.fsum(xo)
    for prec, accel in ((gpu.F64, 0), (gpu.F64, 1), (gpu.F32, 1)):
        x, r = A.pagerank_host(beta=0.85, tol=1e-11, max_iter=5000, mode=gpu.PR_DANGLING, precision=prec, accel=accel)
        # ||x - G(x)||_1 < tol: within tol / (1 - beta) of the fixed point
        assert r.converged and np.abs(x - xo).sum() <= 1e-11 / 0.15 + 1e-12


@pytest.mark.parametrize("rows", [255, 256, 257, 511, 513, 4000])
def test_batch_members_with_a_copy_of_their_own(gpu, rows):
    """Members around the size from which a batch builds their ELL-layout
    copy: the one-thread-per-row product's bits, also after new values, and
    the handle's own products are as before."""
    rng = np.random.default_rng(rows)
    n_col, c = rows + 3, 9
    rp = (np.arange(rows + 1) * c).astype(np.int32)
    ci = rng.integers(0, n_col, rows * c).astype(np.int32)
    va = rng.uniform(-1, 1, rows * c)
    A = gpu.DeviceMatrix.csr(rows + 2, n_col, rp, ci, va, stores=gpu.STORE_F64 | gpu.STORE_F32, rows=rows)
    A.tune(gpu.TUNE_SHORT_ROWS, 0)
    held = A.info().device_bytes
    B = gpu.Batch([A])
    slots = (rows + 31) // 32 * 32 * c  # rows are padded to a multiple of 32, by at most 1/32 of the entries
    copied = rows >= 256 and slots <= rows * c + rows * c // 32
    assert (A.info().device_bytes > held) == copied and A.info().slices == 0
    for store, tdt in ((gpu.F64, torch.float64), (gpu.F32, torch.float32)):
        x = torch.rand(n_col, dtype=tdt, device="cuda")
        y, ref = (torch.full((rows + 2,), 7.0, dtype=tdt, device="cuda") for _ in range(2))
        B.bind(store, [x.data_ptr()], [y.data_ptr()])
        for new in (False, True):
            if new:
                A.set_values(gpu.F64, torch.from_numpy(rng.uniform(-1, 1, rows * c)).cuda().data_ptr())
            y.fill_(7.0)
            B.spmv()
            A.spmv_ex(store, gpu.F64 if store == gpu.F64 else gpu.F32, x.data_ptr(),
                      gpu.F64 if store == gpu.F64 else gpu.F32, ref.data_ptr())
            assert torch.equal(y, ref)


@pytest.mark.parametrize("count", [5, 6, 16])
def test_batch_items_and_grid_by_row_count(gpu, count):
    """Both item spans and both default grids: each member's rows carry the
    bits of its own one-thread-per-row product."""
    rng = np.random.default_rng(count)
    rows, c = 60001, 5
    rp = (np.arange(rows + 1) * c).astype(np.int32)
    mats, xs, ys = [], [], []
    for _ in range(count):
        ci = rng.integers(0, rows, rows * c).astype(np.int32)
        A = gpu.DeviceMatrix.csr(rows, rows, rp, ci, rng.uniform(-1, 1, rows * c), stores=gpu.STORE_F64, rows=rows)
        A.tune(gpu.TUNE_SHORT_ROWS, 0)
        mats.append(A)
        xs.append(torch.rand(rows, dtype=torch.float64, device="cuda"))
        ys.append(torch.full((rows,), 7.0, dtype=torch.float64, device="cuda"))
    B = gpu.Batch(mats)
    B.bind(gpu.F64, [x.data_ptr() for x in xs], [y.data_ptr() for y in ys])
    B.spmv()
    ref = torch.empty(rows, dtype=torch.float64, device="cuda")
    for A, x, y in zip(mats, xs, ys):
        A.spmv_ex(gpu.F64, gpu.F64, x.data_ptr(), gpu.F64, ref.data_ptr())
        assert torch.equal(y, ref)

"""DENSE products at the edges of the rule that gives many rows of few columns four rows a
warp: row counts and column counts on both sides, rows that are no multiple of
four or of a block's 32, columns below, at and above a step of 32, x on and off 16
bytes, every store.

Bound: a sum of c products, each rounded once and added in any order, is within
(c + 1) u sum|a x| of exact, on both sides (u = 2^-53, 2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,cols", [(9727, 64), (9728, 64), (9729, 1), (9731, 33), (9728, 192), (9728, 193), (16383, 320), (16384, 320),
                                       (16384, 321), (5, 192), (1001, 193), (9728, 288), (9728, 289), (3, 7), (32767, 100), (32768, 100), (32770, 130), (32768, 512), (32769, 513), (32768, 400), (32768, 408),
                                       (9733, 1500), (9728, 2047), (9729, 2049), (300001, 3), (100003, 31)])
def test_rows_of_few_columns(gpu, rows, cols):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    a = torch.rand((rows, cols), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    a = a.bfloat16().double()  # every store holds the same values
    x = torch.rand(cols + 1, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    A = gpu.DeviceMatrix.dense(rows, cols, rows, cols, a.cpu().numpy().ravel(),
                               stores=gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16)
    for store, vt, dt, u in ((gpu.F64, gpu.F64, torch.float64, 2.0 ** -53),
                             (gpu.F32, gpu.F32, torch.float32, 2.0 ** -24),
                             (gpu.BF16, gpu.F32, torch.float32, 2.0 ** -24)):
        for off in (0, 1):
            xs = x.to(dt)[off:off + cols].clone() if off == 0 else x.to(dt)[off:off + cols]
            y = torch.full((rows + 3,), 7.0, dtype=dt, device="cuda")
            A.spmv_ex(store, vt, xs.data_ptr(), vt, y.data_ptr())
            want = a @ xs.double()
            scale = a.abs() @ xs.double().abs()
            err = (y[:rows].double() - want).abs()
            assert bool((err <= 2 * (cols + 2) * u * scale).all()), (store, off, float((err / scale).max()))
            assert bool((y[rows:] == 7.0).all())

"""Tensor-core DENSE products whose rows, or whose vectors, do not start on 16 bytes and
are copied with padding first: widths on both sides of the copy's rule (64
elements), and narrow ones, whose copy runs over the row ends.  Against FP64 of the
values as the tensor cores take them.

Bound: FP32 operands are rounded to TF32 (10 bits: 2^-11 each), BF16 ones are exact
here but for X (2^-9); products add in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,c", [(70001, 3), (3000, 31), (20000, 63), (20001, 65), (513, 255), (513, 257), (999, 130), (4096, 1), (777, 511)])
@pytest.mark.parametrize("k", [8, 33])
def test_padded_copies(gpu, m, c, k):
    g = torch.Generator(device="cuda").manual_seed(m + c + k)
    a = (torch.rand((m, c), dtype=torch.float64, device="cuda", generator=g) * 2 - 1).bfloat16().double()
    x = torch.rand((k, c), dtype=torch.float32, device="cuda", generator=g) * 2 - 1
    A = gpu.DeviceMatrix.dense(m, c, m, c, a.cpu().numpy().ravel(), stores=gpu.STORE_F64 | gpu.STORE_F32 | gpu.STORE_BF16)
    want, scale = x.double() @ a.T, x.double().abs() @ a.abs().T
    for store, rel in ((gpu.F32, 2.0 ** -10), (gpu.BF16, 2.0 ** -8)):
        y = torch.full((k, m + 5), 7.0, dtype=torch.float32, device="cuda")
        A.dense_spmm(store, k, x.data_ptr(), c, y.data_ptr(), m + 5)
        assert A.device_status() == 0
        err = (y[:, :m].double() - want).abs()
        assert bool((err <= (rel + (c + 2) * 2.0 ** -23) * scale).all()), float((err / scale).max())
        assert bool((y[:, m:] == 7.0).all())

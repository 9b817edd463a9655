"""The values gradient where rows with entries lie far apart: runs of empty rows
inside a segment of entries, before and after it, rows of one entry at any
distance, one long row among them.  Every gradient is one rounded product of
(scale a[row]) and b[col]: equal to numpy's bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def gaps(kind, rng):
    if kind == "run":                # a run of a million empty rows in the middle of a segment
        ln = rng.integers(0, 5, 4000)
        ln[10] = 100
        return np.concatenate([ln[:1777], np.zeros(1_000_000, int), ln[1777:]])
    if kind == "ends":               # empty rows first and last, one entry left for the last segment
        ln = np.concatenate([np.zeros(70_000, int), np.full(1, 128 * 3), np.zeros(90_000, int), np.full(1, 1),
                             np.zeros(50_000, int)])
        return ln
    if kind == "mixed":              # dense and sparse stretches in turn
        ln = rng.integers(0, 3, 300_000)
        for a in range(0, 300_000, 7001):
            ln[a:a + 5000] = rng.random(5000) < 0.004
        ln[[5, 150_000, 299_999]] = [700, 33, 129]
        return ln
    every = int(kind)                # one entry every `every` rows
    ln = np.zeros(200_000, int)
    ln[::every] = 1
    ln[77] = 100
    return ln


@pytest.mark.parametrize("kind", ["run", "ends", "mixed", "1", "2", "16", "31", "32", "33", "64", "1000"])
@pytest.mark.parametrize("dt", ["F64", "F32"])
def test_gradient_bits(gpu, kind, dt):
    rng = np.random.default_rng(9)
    ln = gaps(kind, rng)
    n = ln.size
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    A = gpu.DeviceMatrix.csr(n, n, rp, ci, np.ones(rp[-1]))
    t = np.float64 if dt == "F64" else np.float32
    a, b, scale = rng.uniform(-1, 1, n).astype(t), rng.uniform(-1, 1, n).astype(t), t(0.85)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.full((int(rp[-1]) + 32,), 7.0, dtype=ta.dtype, device="cuda")
    A.grad_values(getattr(gpu, dt), ta.data_ptr(), tb.data_ptr(), float(scale), out.data_ptr())
    got = out.cpu().numpy()
    assert np.array_equal(got[:rp[-1]], (scale * a)[np.repeat(np.arange(n), ln)] * b[ci])
    assert np.all(got[rp[-1]:] == 7.0)


def test_a_run_of_empty_rows_costs_no_walk(gpu):
    """4 million empty rows between two entries: walked by one warp they took 54 ms,
    against 13 us without them.  Event times; the bound leaves 40 times that."""
    rng = np.random.default_rng(3)
    ln = rng.integers(0, 5, 4000)
    ln[10] = 100
    ln = np.concatenate([ln[:2000], np.zeros(4_000_000, int), ln[2000:]])
    n = ln.size
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    A = gpu.DeviceMatrix.csr(n, n, rp, rng.integers(0, n, rp[-1]).astype(np.int32), np.ones(rp[-1]))
    a, b = torch.ones(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    out = torch.empty(int(rp[-1]), dtype=torch.float64, device="cuda")
    times = []
    for _ in range(8):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        A.grad_values(gpu.F64, a.data_ptr(), b.data_ptr(), 1.0, out.data_ptr())
        e.record()
        torch.cuda.synchronize()
        times.append(s.elapsed_time(e))
    assert sorted(times)[3] < 0.5, times

"""Rows that the tensor-core pass hands to the exact FP32 scan (nearly equal centers: every center is
a candidate) get the FP32 path's labels and costs: list lengths around four rows, the 2048 that the
short-list kernel takes and past it, centers around a thread block, through a single pass (length
known on the host) and through the device loop (length known on the device)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, k):
    rng = np.random.default_rng(n * 3 + d + k)
    base = rng.normal(size=d).astype(np.float32) * 4
    C = (base + rng.normal(size=(k, d)) * 1e-3).astype(np.float32)
    C[k - 1] = C[2]  # a tie: the lower index wins
    X = (base + rng.normal(size=(n, d)) * 1e-3).astype(np.float32)
    far = (rng.normal(size=(3000, d)) * 0.01 + base + 50).astype(np.float32)  # settled rows
    return np.concatenate([X, far]), np.concatenate([C, far[:1]])


@pytest.mark.parametrize("n,d,k", [(1, 128, 40), (3, 20, 127), (4, 64, 128), (5, 33, 129), (2047, 16, 60),
                                   (2048, 128, 40), (2049, 64, 40), (6000, 32, 300)])
def test_rescanned_rows_equal_fp32(n, d, k):
    import minicore_gb300 as mc
    X, C = _data(n, d, k)
    out = {}
    for precision in ("fp32", "bf16"):
        job = mc.Job(X, C, msr=2, prior=0.0, precision=precision)
        job.assign()
        a, c = np.empty(len(X), np.uint32), np.empty(len(X), np.float64)
        job.read(None, a, c)
        job.run(eps=0.0, maxiter=3)
        cen, a2, c2 = np.empty(C.shape, np.float32), np.empty(len(X), np.uint32), np.empty(len(X), np.float64)
        job.read(cen, a2, c2)
        job.close()
        out[precision] = (a, c, cen, a2, c2)
    for x, y in zip(out["fp32"], out["bf16"]):
        assert np.array_equal(x, y)

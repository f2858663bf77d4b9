"""Dense L1 medians over columns with infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [40, 41])
def test_medians_with_infinities_and_nan(m):
    """Rows that are infinite or NaN fall to center 0; the median orders them as the values' bits do
    (-inf first, NaN last)."""
    import minicore_gb300 as mc
    rng = np.random.default_rng(m)
    d = 9
    A = rng.integers(-3, 4, (m, d)).astype(np.float32)
    for col in range(d):  # none to all of the rows at one end
        A[:min(m, 5 * col), col] = [np.inf, -np.inf, np.nan][col % 3]
    B = rng.integers(-3, 4, (30, d)).astype(np.float32) + np.float32(1000.0)
    X = np.concatenate([A, B])
    C = np.stack([np.zeros(d, np.float32), np.full(d, 1000.0, np.float32)])
    job = mc.Job(X, C, msr=0)
    job.assign()
    job.lloyd_step()
    got = np.empty_like(C)
    job.read(got, None, None)
    job.close()
    for c, V in enumerate((A, B)):
        v = np.sort(V, axis=0)
        lo, hi = v[(len(V) - 1) // 2], v[len(V) // 2]
        with np.errstate(invalid="ignore"):
            want = hi if len(V) & 1 else np.float32(0.5) * (lo + hi)
        assert np.array_equal(got[c], want, equal_nan=True)

"""Dense L1 medians of clusters whose keys do not fit shared memory, beside small ones, odd and even, with
ties, columns past a CTA's eight and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(30000, 5, 2, 1), (20001, 9000, 64, 3), (7000, 7001, 6900, 6801)])
@pytest.mark.parametrize("d", [1, 8, 19])
def test_large_clusters(sizes, d):
    import minicore_gb300 as mc
    rng = np.random.default_rng(sum(sizes) + d)
    mu = np.array([-1000.0, 0.0, 1000.0, 2000.0], np.float32)
    lab = np.repeat(np.arange(4), sizes)
    rng.shuffle(lab)
    X = (mu[lab][:, None] + rng.integers(-40, 41, (lab.size, d)) * np.float32(0.5)).astype(np.float32)
    if d > 1:  # NaN distances fall to center 0
        X[np.flatnonzero(lab == 0)[:sizes[0] // 3], d - 1] = np.nan
        X[np.flatnonzero(lab == 0)[-7:], 0] = np.inf
    C = np.repeat(mu[:, None], d, 1)
    job = mc.Job(X, C, msr=0)
    job.assign()
    job.lloyd_step()
    got = np.empty_like(C)
    job.read(got, None, None)
    job.close()
    for c in range(4):
        v = np.sort(X[lab == c], axis=0)
        m = v.shape[0]
        lo, hi = v[(m - 1) // 2], v[m // 2]
        assert np.array_equal(got[c], hi if m & 1 else np.float32(0.5) * (lo + hi), equal_nan=True)

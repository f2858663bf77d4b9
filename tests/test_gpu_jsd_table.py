"""JSD over grouped count rows: the zero-entry table formed with and without the centers' logarithms
beforehand (from 2,000,000 terms on) is the same, so centers assigned alone have the distances that they
have among many."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,per", [(1100, 30), (3000, 60)])
def test_few_centers_equal_many(d, per):
    import minicore_gb300 as mc
    rng = np.random.default_rng(d)
    n, groups = 600, 6
    rows = [np.sort(rng.choice(d, per * 10 + g, replace=False)) for g in range(groups) for _ in range(n // groups)]
    ip = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    X = sp.csr_matrix((np.ones(ip[-1], np.float32), np.concatenate(rows).astype(np.int32), ip), shape=(n, d))
    k = 2000000 // (groups * d) + 1
    C = (rng.random((k, d)) * (rng.random((k, d)) < 0.6)).astype(np.float32)
    many = mc.cmp(X, C, msr=4, prior=1.0)
    for c in (0, 3, k - 5):
        assert np.array_equal(mc.cmp(X, C[c:c + 5], msr=4, prior=1.0), many[:, c:c + 5])

"""JSD over wide CSR count rows: the pass by groups of rows with equal zero-entry values gives, bit
for bit, what the gather kernel gives, which takes the same rows when there are fewer than eight per
group.  Groups cover more than one and two slabs, less than a slab, a single row (no table) and rows
without entries; center counts cover one to three passes of 64, odd and full; the column count
leaves a partial band and none."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mc():
    import minicore_gb300 as m
    return m


def _assign(mc, X, C):
    from minicore_gb300 import _lib
    M = mc._MatrixArg(X)
    asn = np.empty(M.n, np.uint32)
    costs = np.empty(M.n, np.float64)
    _lib.check(_lib.load().mc_assign(mc.default_context().handle, M.ref, mc._p(C), C.shape[0], 4, 1.0, 0,
                                     mc._p(asn), mc._p(costs)))
    return asn, costs


@pytest.mark.parametrize("d", [2100, 2304])
@pytest.mark.parametrize("k", [33, 50, 64, 97, 128, 161])
def test_groups_equal_gather(mc, d, k):
    rng = np.random.default_rng(d + k)
    total = np.repeat([1200, 1290, 1301, 1340, 0], [130, 200, 37, 1, 9])
    rng.shuffle(total)
    rows = []
    for s in total:
        twos = int(rng.integers(0, 60)) if s else 0
        r = np.zeros(d, np.float32)
        cols = rng.choice(d, int(s) - twos, replace=False)
        r[cols] = 1.0
        r[cols[:twos]] = 2.0
        rows.append(r)
    D = np.stack(rows)
    X = sp.csr_matrix(D)
    X.sort_indices()
    C = (rng.random((k, d)) * (rng.random((k, d)) < 0.7) * 3).astype(np.float32)
    C[: k // 2] += D[rng.choice(len(D), k // 2)]
    mc.autotune(False)
    try:
        asn, costs = _assign(mc, X, C)
        for part in range(2):
            ids = np.concatenate([np.flatnonzero(total == s)[7 * part:7 * part + 7] for s in np.unique(total)])
            a0, c0 = _assign(mc, X[ids], C)
            assert np.array_equal(asn[ids], a0)
            assert np.array_equal(costs[ids], c0)
    finally:
        mc.autotune(True)

"""CSR row sums (the prior setup reads them): whole-number rows are added as integers, other rows
entry by entry in FP64; both equal the oracle's sequential sum, so the distances do too.  The
structure check must still refuse malformed rows."""
import numpy as np
import pytest

sp = pytest.importorskip("scipy.sparse")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000])
def test_csr_row_sums_feed_exact_distances(n):
    import minicore_gb300 as mc
    import oracle
    rng = np.random.default_rng(n)
    d = 700
    rows = []
    for i in range(n):
        m = int(rng.integers(0, 140)) if i % 5 else (0 if i % 2 else 33)
        c = np.sort(rng.choice(d, m, replace=False))
        kind = i % 4
        if kind == 0:
            v = rng.integers(1, 9, m).astype(np.float32)                      # counts
        elif kind == 1:
            v = rng.integers(1, 9, m).astype(np.float32) * np.float32(2.0) ** 28  # large whole numbers
        elif kind == 2:
            v = (rng.random(m) * 5).astype(np.float32)                        # fractions
        else:
            v = rng.integers(1, 9, m).astype(np.float32)
            if m:
                v[-1] = np.float32(0.5)                                       # one fraction at the end
        rows.append(sp.csr_matrix((v, c, [0, m]), shape=(1, d)))
    X = sp.vstack(rows).tocsr().astype(np.float32)
    X.sort_indices()
    C = rng.integers(0, 5, (3, d)).astype(np.float32) + 1.0
    # Hellinger's pair scalars divide by the row sum: relative 1e-4 is the CSR measures' bar
    for msr in (5, 6):
        D = mc.cmp(X, C, msr=msr, prior=1.0)
        E = np.stack([oracle.assign(X, C[j:j + 1], msr, 1.0)[1] for j in range(3)], 1)
        assert np.allclose(D, E, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("bad,what", [("order", "strictly increasing"), ("range", "< ncols"), ("ptr", "nondecreasing")])
@pytest.mark.parametrize("row", [0, 40, 99])
def test_malformed_csr_is_refused(bad, what, row):
    import minicore_gb300 as mc
    n, d, m = 100, 500, 40
    idx = np.tile(np.arange(0, 2 * m, 2, dtype=np.uint32), n)
    ptr = np.arange(0, n * m + 1, m).astype(np.uint64)
    if bad == "order":
        idx[row * m + 33] = idx[row * m + 32]
    elif bad == "range":
        idx[row * m + m - 1] = d
    elif row:
        ptr[row] = ptr[row - 1] - 1 if row > 1 else 0
    else:
        ptr[1] = n * m + 5
    X = mc.CSparseMatrix(data=np.ones(n * m, np.float32), indices=idx, indptr=ptr, shape=(n, d))
    with pytest.raises(ValueError):
        mc.kmeanspp(X, 3, msr=5, prior=1.0, seed=2)

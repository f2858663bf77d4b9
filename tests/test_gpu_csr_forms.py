"""CSR rows long enough for a warp each: row sums of whole numbers and of others, and the structure check."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def test_long_rows_have_the_sums_of_short_ones():
    """The same rows beside many empty ones (few entries a row on average: a thread per row) give the
    same distances bit for bit: the pair scalars read the sums."""
    import minicore_gb300 as mc
    rng = np.random.default_rng(2)
    d = 4000
    rows = []
    for i in range(36):
        m = int(rng.integers(500, 3000)) if i % 9 else (0, 1, 31, 33)[i // 9]
        v = rng.integers(1, 9, m).astype(np.float32)
        if i % 4 == 1:
            v *= np.float32(2.0) ** 28                    # 2^31 and above among them
        elif i % 4 == 2:
            v = (rng.random(m) * 5).astype(np.float32)
        elif i % 4 == 3 and m:
            v[[-1, m // 2][i // 4 % 2]] = 0.5             # one fraction, past the first 32 entries or last
        if i == 20:
            v[40] = np.nan
        if i == 24:
            v[3] = np.inf
        rows.append(sp.csr_matrix((v, np.sort(rng.choice(d, m, replace=False)), [0, m]), shape=(1, d)))
    X = sp.vstack(rows).tocsr().astype(np.float32)
    assert X.nnz >= 512 * X.shape[0]
    more = sp.vstack([X, sp.csr_matrix((400, d), dtype=np.float32)]).tocsr()
    C = rng.integers(0, 5, (3, d)).astype(np.float32) + 1.0
    for msr in (5, 6):
        D = mc.cmp(X, C, msr=msr, prior=1.0)
        E = mc.cmp(more, C, msr=msr, prior=1.0)[:X.shape[0]]
        assert np.array_equal(D, E, equal_nan=True)


@pytest.mark.parametrize("m", [159, 160, 300])
@pytest.mark.parametrize("bad", ["order", "range", "ptr"])
@pytest.mark.parametrize("row", [0, 40, 99])
def test_malformed_rows_are_refused(bad, row, m):
    import minicore_gb300 as mc
    n, d = 100, 1000
    idx = np.tile(np.arange(0, 2 * m, 2, dtype=np.uint32), n)
    ptr = np.arange(0, n * m + 1, m).astype(np.uint64)
    if bad == "order":
        idx[row * m + 129] = idx[row * m + 128]
    elif bad == "range":
        idx[row * m + m - 1] = d
    elif row:
        ptr[row] = ptr[row - 1] - 1 if row > 1 else 0
    else:
        ptr[1] = n * m + 5
    X = mc.CSparseMatrix(data=np.ones(n * m, np.float32), indices=idx, indptr=ptr, shape=(n, d))
    with pytest.raises(ValueError):
        mc.kmeanspp(X, 3, msr=5, prior=1.0, seed=2)

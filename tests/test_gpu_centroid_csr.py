"""Centroid update over CSR rows against the documented order of its sums, bit for bit: rows of
a cluster ascending in chunks of 4096, per chunk and column a compensated float sum (weighted:
an FP64 fma sum), chunk sums added in FP64 in order, divided by the count (weight)."""
import numpy as np
import pytest

sp = pytest.importorskip("scipy.sparse")
pytestmark = pytest.mark.gpu


def _rows(n, d, avg, seed, dense_rows=(), cluster_cols=0):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 2 * avg + 1, n)
    lens[rng.integers(0, n, n // 50)] = 0
    lens[list(dense_rows)] = d
    idx, ptr = [], [0]
    for i in range(n):
        m = min(int(lens[i]), d)
        if cluster_cols and i % 7 == 0 and m:  # this row's entries side by side: one band takes them
            b = int(rng.integers(0, d - m + 1))
            c = np.arange(b, b + m)
        else:
            c = np.sort(rng.choice(d, m, replace=False))
        idx.append(c)
        ptr.append(ptr[-1] + m)
    idx = np.concatenate(idx).astype(np.int32)
    # values over six decades: float sums that round
    val = (rng.normal(size=idx.size) * 10.0 ** rng.integers(-3, 4, idx.size)).astype(np.float32)
    return sp.csr_matrix((val, idx, np.asarray(ptr)), shape=(n, d))


def _two_sum(s, e, x):
    t = s + x
    bp = t - s
    return t, e + ((s - (t - bp)) + (x - bp))


def _expected(X, asn, C, w):
    out = C.copy()
    for c in range(C.shape[0]):
        rows = np.nonzero(asn == c)[0]
        if rows.size == 0:
            continue
        if rows.size == 1:
            out[c] = X[rows[0]].toarray().ravel()
            continue
        S, den = None, None
        for b in range(0, rows.size, 4096):
            ch = rows[b:b + 4096]
            if w is None:
                s = np.zeros(X.shape[1], np.float32)
                e = np.zeros(X.shape[1], np.float32)
                for r in ch:
                    j = X.indices[X.indptr[r]:X.indptr[r + 1]]
                    s[j], e[j] = _two_sum(s[j], e[j], X.data[X.indptr[r]:X.indptr[r + 1]])
                p, q = s.astype(np.float64) + e.astype(np.float64), float(ch.size)
            else:
                # weights are powers of two: the fma's product is exact, so it is a plain sum
                p, q = np.zeros(X.shape[1]), 0.0
                for r in ch:
                    j = X.indices[X.indptr[r]:X.indptr[r + 1]]
                    p[j] = p[j] + w[r] * X.data[X.indptr[r]:X.indptr[r + 1]].astype(np.float64)
                    q += w[r]
            S, den = (p, q) if S is None else (S + p, den + q)
        out[c] = (S / (float(rows.size) if w is None else den)).astype(np.float32)
    return out


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,d,avg,k,dense,cluster", [
    (9000, 600, 5, 2, 0, 0),       # short rows: two chunks per cluster, two 512-column bands
    (1500, 2048, 20, 9, 0, 0),     # short rows: four full bands, a partial last batch
    (3000, 512, 6, 3, 60, 0),      # a batch with more entries than slots (dense tile)
    (700, 70, 1, 40, 0, 0),        # few rows per cluster, single rows and empty ones
    (6000, 3000, 200, 3, 0, 1),    # bands of 512 columns, a ragged last one; long parts (> 64)
    (4700, 20000, 300, 1, 0, 1),   # one cluster, two chunks, ten bands of 2048
    (900, 2100, 40, 4, 3, 0),      # 2048-column bands, rows with every column
    (500, 130, 60, 30, 0, 0),      # 128-column bands
])
def test_csr_centroids_follow_the_documented_order(n, d, avg, k, dense, cluster, weighted):
    import minicore_gb300 as mc
    X = _rows(n, d, avg, n + d, range(100, 100 + dense), cluster)
    rng = np.random.default_rng(k)
    C = np.asarray(X[rng.choice(n, k, replace=False)].toarray(), np.float32)
    w = 2.0 ** rng.integers(-3, 4, n) if weighted else None
    job = mc.Job(X, C, msr=2, weights=w, seed=3)
    job.assign()
    asn = np.empty(n, np.uint32)
    job.read(None, asn, None)
    if (np.bincount(asn, minlength=k) == 0).any():  # no D^2 restart in this comparison
        keep = np.unique(asn)
        job.close()
        C = C[keep]
        job = mc.Job(X, C, msr=2, weights=w, seed=3)
        job.assign()
        job.read(None, asn, None)
    for _ in range(2):  # the second update reuses the job's band offsets
        got = np.empty_like(C)
        assert not job.lloyd_step()
        job.read(got, None, None)
        want = _expected(X, asn, C, w)
        assert np.array_equal(got, want)
        C = got
        job.read(None, asn, None)
        if (np.bincount(asn, minlength=C.shape[0]) == 0).any():
            break
    job.close()

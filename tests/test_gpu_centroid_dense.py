"""Centroid update over dense rows against the documented order of its sums, bit for bit (rows of
a cluster ascending in chunks of 256, a compensated float sum per chunk and column; weighted: FP64
fma sums; chunk sums added in FP64): vector widths of 4, 2 and 1 columns per lane, partial lanes,
chunk counts around 256 rows and batches around 8 and 32 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expected(X, asn, C, w):
    out = C.copy()
    for c in range(C.shape[0]):
        rows = np.nonzero(asn == c)[0]
        if rows.size <= 1:
            if rows.size:
                out[c] = X[rows[0]]
            continue
        S, den = None, None
        for b in range(0, rows.size, 256):
            ch = rows[b:b + 256]
            if w is None:
                s, e = np.zeros(X.shape[1], np.float32), np.zeros(X.shape[1], np.float32)
                for r in ch:
                    t = s + X[r]
                    bp = t - s
                    e = e + ((s - (t - bp)) + (X[r] - bp))
                    s = t
                p, q = s.astype(np.float64) + e.astype(np.float64), float(ch.size)
            else:  # weights are powers of two: the fma's product is exact
                p, q = np.zeros(X.shape[1]), 0.0
                for r in ch:
                    p = p + w[r] * X[r].astype(np.float64)
                    q += w[r]
            S, den = (p, q) if S is None else (S + p, den + q)
        out[c] = (S / (float(rows.size) if w is None else den)).astype(np.float32)
    return out


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,d,k", [(700, 128, 2), (257, 100, 1), (256, 96, 1), (255, 50, 1), (40, 48, 3), (2000, 33, 6),
                                   (600, 3, 2), (520, 260, 2), (33, 130, 1), (9, 64, 1), (900, 47, 30)])
def test_dense_centroids_follow_the_documented_order(n, d, k, weighted):
    import minicore_gb300 as mc
    rng = np.random.default_rng(n * d + k)
    X = (rng.normal(size=(n, d)) * 10.0 ** rng.integers(-3, 4, (n, 1))).astype(np.float32)
    C = X[rng.choice(n, k, replace=False)].copy()
    w = 2.0 ** rng.integers(-3, 4, n) if weighted else None
    job = mc.Job(X, C, msr=2, weights=w, seed=3)
    job.assign()
    asn, got = np.empty(n, np.uint32), np.empty_like(C)
    job.read(None, asn, None)
    assert not job.lloyd_step()
    job.read(got, None, None)
    job.close()
    assert np.array_equal(got, _expected(X, asn, C, w))

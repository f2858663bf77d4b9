"""Dense L1 with prior 0: assignments and medians equal the oracle's bit for bit where the pair's
tiny prior cannot change a term (ordinary values) and where it can (magnitudes next to it), and for
clusters below and above what a median's CTA holds in shared memory, odd and even, tied and signed.
Soft clustering's center sums at the edges of their tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e-36, 1e-41])
@pytest.mark.parametrize("n,d,k", [(130, 17, 5), (300, 70, 70)])
def test_l1_assignment_with_prior_zero(scale, n, d, k):
    import minicore_gb300 as mc
    import oracle
    rng = np.random.default_rng(n + d)
    X = rng.integers(0, 5, (n, d)).astype(np.float32)
    X[::3] *= np.float32(scale)  # zeros, ordinary values and values of this magnitude together
    X[0] = 0
    C = X[rng.choice(n, k, replace=False)].copy()
    C[0, ::2] += np.float32(3.0)
    job = mc.Job(X, C, msr=0, prior=0.0)
    job.assign()
    asn, cost = np.empty(n, np.uint32), np.empty(n, np.float64)
    job.read(None, asn, cost)
    job.close()
    oasn, ocost = oracle.assign(X, C, 0, 0.0)
    assert np.array_equal(asn, oasn)
    assert np.array_equal(cost, ocost)


@pytest.mark.parametrize("sizes", [(1, 2, 3, 4), (31, 32, 33, 64), (700, 10, 11, 12), (9000, 5, 8000, 6), (257, 256, 255, 254)])
@pytest.mark.parametrize("d", [1, 8, 13])
def test_dense_medians(sizes, d):
    import minicore_gb300 as mc
    rng = np.random.default_rng(sum(sizes) + d)
    mu = np.array([-1000.0, 0.0, 1000.0, 2000.0], np.float32)
    lab = np.repeat(np.arange(4), sizes)
    rng.shuffle(lab)
    X = (mu[lab][:, None] + rng.integers(-3, 4, (lab.size, d)) * np.float32(0.5)).astype(np.float32)
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
        assert np.array_equal(got[c], hi if m & 1 else np.float32(0.5) * (lo + hi))


@pytest.mark.parametrize("n,d,k,weighted", [(1, 3, 1, False), (255, 32, 4, False), (257, 33, 33, True), (1300, 70, 100, False),
                                            (9000, 5, 20, True), (520, 31, 400, False)])
def test_soft_clustering_edges(n, d, k, weighted):
    import minicore_gb300 as mc
    import oracle
    rng = np.random.default_rng(n + d + k)
    X = (rng.normal(size=(n, d)) + rng.integers(0, 4, (n, 1)) * 2.0).astype(np.float32)
    C = X[rng.choice(n, k, replace=k > n)].copy() + rng.normal(size=(k, d)).astype(np.float32) * np.float32(0.1)
    w = rng.uniform(0.5, 2.0, n) if weighted else None
    r = mc.scluster(X, C, msr=2, temp=0.5, maxiter=2, weights=w)
    o = oracle.scluster(X, C, 2, 0.0, temp=0.5, maxiter=2, weights=w)
    assert r["numiter"] == o["numiter"]
    assert np.allclose(r["centers"], o["centers"], rtol=1e-4, atol=1e-5)
    assert np.allclose(r["asn"], o["asn"], atol=1e-5)


@pytest.mark.parametrize("rows,centers", [(1.0, 1.0), (1e-41, 1.0), (1.0, 1e-41)])
@pytest.mark.parametrize("n,d,k", [(38912, 80, 33), (38913, 80, 33), (50001, 41, 64), (100001, 15, 66)])
def test_l1_assignment_of_many_rows(rows, centers, n, d, k):
    """Sizes from which plain differences have a kernel of their own: taken, ruled out by the rows and
    ruled out by the centers alone (the pair kernel's CTAs then walk several tiles each)."""
    import minicore_gb300 as mc
    import oracle
    rng = np.random.default_rng(n + k)
    X = rng.integers(0, 5, (n, d)).astype(np.float32)
    C = X[rng.choice(n, k, replace=False)].copy()
    X[::3] *= np.float32(rows)
    C[::2] *= np.float32(centers)
    C[0, ::2] += np.float32(3.0)
    job = mc.Job(X, C, msr=0, prior=0.0)
    job.assign()
    asn, cost = np.empty(n, np.uint32), np.empty(n, np.float64)
    job.read(None, asn, cost)
    job.close()
    oasn, ocost = oracle.assign(X, C, 0, 0.0)
    assert np.array_equal(asn, oasn)
    assert np.array_equal(cost, ocost)

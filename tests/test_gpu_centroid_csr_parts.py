"""Centroid sums of short CSR rows whose batches of 512 have more entries than are ordered at once: halves
and quarters of a batch, and a quarter that has more still."""
import numpy as np
import pytest

pytest.importorskip("scipy.sparse")
from test_gpu_centroid_csr import _expected, _rows  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,d,avg,k,dense", [(5000, 171, 20, 2, 0), (1100, 400, 29, 1, 0), (3000, 512, 20, 3, 60),
                                             (2000, 1030, 31, 2, 0), (300, 150, 31, 1, 0)])
def test_batches_in_parts(n, d, avg, k, dense, weighted):
    import minicore_gb300 as mc
    X = _rows(n, d, avg, n + d, range(100, 100 + dense))
    assert X.nnz < 32 * n
    rng = np.random.default_rng(k)
    C = np.asarray(X[rng.choice(n, k, replace=False)].toarray(), np.float32)
    w = 2.0 ** rng.integers(-3, 4, n) if weighted else None
    job = mc.Job(X, C, msr=2, weights=w, seed=3)
    job.assign()
    asn = np.empty(n, np.uint32)
    job.read(None, asn, None)
    assert (np.bincount(asn, minlength=k) > 0).all()
    got = np.empty_like(C)
    assert not job.lloyd_step()
    job.read(got, None, None)
    job.close()
    assert np.array_equal(got, _expected(X, asn, C, w))

"""Counting sort whose key scan also writes the bucket and chunk starts: key counts around one key
per thread, the largest that is scanned in the same launch and the first that is not, row counts
around a tile; two passes, so that a second sort reuses the first one's scratch.  The centroid means
and the order of equal keys are the oracle's (exact: sums are in the canonical order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (511, 2), (513, 255), (2000, 256), (3000, 257), (9000, 4096), (9000, 4097)])
def test_means_after_sort(n, k):
    import minicore_gb300 as mc
    rng = np.random.default_rng(n + k)
    d = 3
    k = min(k, n)
    C = (np.arange(k)[:, None] * 16 + rng.normal(size=(k, d))).astype(np.float32)
    lab = np.concatenate([np.arange(k), rng.integers(0, k, n - k)])
    rng.shuffle(lab)
    X = (lab[:, None] * 16 + rng.integers(-3, 4, size=(n, d))).astype(np.float32)  # small integers: exact sums
    job = mc.Job(X, C, msr=2, prior=0.0)
    job.assign()
    for _ in range(2):
        assert not job.lloyd_step()  # no center restarted
    centers = np.empty((k, d), np.float32)
    asn = np.empty(n, np.uint32)
    job.read(centers, asn, None)
    job.close()
    assert np.array_equal(asn, lab)
    ref = np.stack([X[lab == c].astype(np.float64).sum(0) / np.count_nonzero(lab == c) for c in range(k)])
    assert np.array_equal(centers, ref.astype(np.float32))


@pytest.mark.parametrize("k", [3, 256, 4096, 4097])
@pytest.mark.parametrize("empty", [False, True])
def test_loop_modes_agree_on_empty_clusters(k, empty):
    """The search for empty clusters, in the sort's last block up to 4096 keys and in a launch of its
    own past them, and the stop rule at the end of the objective's sum: the device loops run as the
    host loop does, with a cluster that is empty from the start (last key) and without."""
    import minicore_gb300 as mc
    rng = np.random.default_rng(k)
    C = (np.arange(k)[:, None] * 16 + np.zeros((1, 3))).astype(np.float32)
    if empty:
        C[k - 1] = -1e6
    m = k - 1 if empty else k
    lab = np.concatenate([np.arange(m), rng.integers(0, m, 2 * m)])
    X = (lab[:, None] * 16 + rng.integers(-3, 4, size=(len(lab), 3))).astype(np.float32)
    out = []
    try:
        for mode in (mc.LOOP_HOST, mc.LOOP_FUSED, mc.LOOP_GRAPH):
            mc.loop_mode(mode)
            job = mc.Job(X, C, msr=2, prior=0.0, seed=3)
            job.run(eps=0.0, maxiter=6)
            cen, asn, cost = np.empty_like(C), np.empty(len(X), np.uint32), np.empty(len(X), np.float64)
            job.read(cen, asn, cost)
            job.close()
            out.append((cen, asn, cost))
    finally:
        mc.loop_mode(mc.LOOP_AUTO)
    for o in out[1:]:
        for x, y in zip(out[0], o):
            assert np.array_equal(x, y)

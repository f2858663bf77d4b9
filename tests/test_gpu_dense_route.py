"""Which kernel takes a dense FP32 assignment, and that every choice gives the same bits: the SQRL2
variants forced through loaded decisions (columns held at once, more than are held, center remainders
of one to three chunks) against the oracle, MKL against the kernel that takes up to 64 centers, L1 at
sizes that are offered the plain form, also with rows it must not take (infinities, NaN)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def mc():
    import minicore_gb300 as m
    yield m
    m.autotune_reset()
    m.autotune(True)


def _assign(mc, X, C, msr, prior=0.0):
    job = mc.Job(X, C, msr=msr, prior=prior)
    job.assign()
    asn, cost = np.empty(len(X), np.uint32), np.empty(len(X), np.float64)
    job.read(None, asn, cost)
    job.close()
    return asn, cost


def _keys(mc):
    return [k for k in mc.autotune_report()["entries"] if k.startswith("dense_sqrl2|dense|")]


@pytest.mark.parametrize("n,d,k", [(700, 192, 65), (300, 193, 80), (257, 401, 130), (130, 48, 97), (129, 112, 200),
                                   (500, 225, 100), (64, 176, 161)])
def test_sqrl2_every_variant_equals_oracle(mc, n, d, k, tmp_path):
    import oracle
    rng = np.random.default_rng(n + d + k)
    X = rng.normal(size=(n, d)).astype(np.float32)
    C = rng.normal(size=(k, d)).astype(np.float32)
    C[k - 1] = C[1]  # a tie: the lower index wins
    X[5, 0], X[9, d - 1] = np.inf, np.nan
    ref = oracle.assign(X, C, 2, 0.0)
    mc.autotune_reset()
    mc.autotune(True)
    _assign(mc, X, C, 2)
    key, = _keys(mc)
    assert len(mc.autotune_report()["entries"][key]["ms"]) == 3
    for v in range(3):
        mc.autotune_reset()
        path = tmp_path / f"v{v}.tsv"
        path.write_text(f"{key}\t{v}\t\n")
        mc.autotune_load(str(path))
        asn, cost = _assign(mc, X, C, 2)
        assert mc.autotune_report()["entries"][key]["variant"] == v
        assert np.array_equal(asn, ref[0]), v
        assert np.array_equal(cost, ref[1], equal_nan=True), v


def test_decisions_of_another_numbering_are_not_taken(mc, tmp_path):
    """A cache file written when 0 was the 8x8 and 1 the 4x4 tile says nothing about today's kernels."""
    rng = np.random.default_rng(3)
    X = rng.normal(size=(20000, 64)).astype(np.float32)
    C = X[:256].copy()
    mc.autotune_reset()
    mc.autotune(True)
    _assign(mc, X, C, 2)
    key, = _keys(mc)
    tag = key.rsplit("|", 1)[1]
    old = f"dense_sqrl2|dense|k256|d2^6|n2^15|{tag}"
    mc.autotune_reset()
    path = tmp_path / "old.tsv"
    path.write_text(f"{old}\t1\t\n")
    mc.autotune_load(str(path))
    _assign(mc, X, C, 2)
    assert sorted(_keys(mc)) == sorted([old, key])  # timed anew


@pytest.mark.parametrize("n,d,k", [(130, 64, 65), (300, 144, 97), (257, 113, 128), (63, 192, 161), (129, 100, 200)])
def test_mkl_equals_the_kernel_of_few_centers(mc, n, d, k):
    rng = np.random.default_rng(n + d + k)
    X = rng.integers(0, 6, (n, d)).astype(np.float32)
    C = rng.integers(0, 6, (k, d)).astype(np.float32) + np.float32(0.25)
    D = mc.cmp(X, C, msr=5, prior=1.0)
    few = np.concatenate([mc.cmp(X, C[c:c + 64], msr=5, prior=1.0) for c in range(0, k, 64)], 1)
    assert np.array_equal(D, few)
    asn, cost = _assign(mc, X, C, 5, 1.0)
    assert np.array_equal(asn, few.argmin(1))
    assert np.array_equal(cost.astype(np.float32), few.min(1))


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("n,d,k", [(38913, 200, 65), (100001, 43, 97), (400001, 20, 10)])
def test_plain_l1_equals_oracle(mc, n, d, k, special):
    import oracle
    rng = np.random.default_rng(n + d)
    X = rng.integers(0, 5, (n, d)).astype(np.float32)
    C = X[rng.choice(n, k, replace=False)] + rng.integers(0, 2, (k, d)).astype(np.float32)
    if special:
        X[7, 3], X[n - 1, d - 1], X[100, 0] = np.inf, -np.inf, np.nan
    asn, cost = _assign(mc, X, C, 0)
    oasn, ocost = oracle.assign(X, C, 0, 0.0)
    assert np.array_equal(asn, oasn)
    assert np.array_equal(cost, ocost, equal_nan=True)

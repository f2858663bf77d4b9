"""Dense FP32 assignment at the edges of its tiles against the oracle's column-by-column sums:
row counts around 64 / 128 rows and past one tile per SM, columns around 16 and past the 192 that
are held at a time, odd columns and unaligned rows (4- and 8-byte copies), and center counts that
leave remainders of 64, 32 and 16.  SQRL2, L1 and Hellinger are exact (no logarithm); MKL takes the
GPU's logf, one ulp of the oracle's: relative 2e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("msr,prior", [(2, 0.0), (0, 0.5), (6, 1.0), (5, 1.0)])  # L1, Hellinger: k_assign_tiled
@pytest.mark.parametrize("n,d,k", [(1, 1, 1), (63, 16, 16), (64, 17, 17), (65, 15, 33), (129, 50, 25), (1000, 100, 49),
                                   (700, 192, 65), (300, 193, 80), (257, 401, 130), (39001, 4, 7), (500, 6, 200)])
def test_dense_assignment_equals_oracle(msr, prior, n, d, k):
    import minicore_gb300 as mc
    import oracle
    rng = np.random.default_rng(n * 7 + d + k)
    if msr in (5, 6):
        X = rng.integers(0, 6, size=(n, d)).astype(np.float32)
        C = rng.integers(0, 6, size=(k, d)).astype(np.float32) + np.float32(0.25)
    else:
        X = rng.normal(size=(n, d)).astype(np.float32)
        C = rng.normal(size=(k, d)).astype(np.float32)
    if k > 3:
        C[k - 1] = C[1]  # a tie: the lower index wins
    if msr == 2 and n > 20:
        X[5, 0] = np.inf
        X[9, d - 1] = np.nan
    job = mc.Job(X, C, msr=msr, prior=prior)
    job.assign()
    asn = np.empty(n, np.uint32)
    cost = np.empty(n, np.float64)
    job.read(None, asn, cost)
    job.close()
    oasn, ocost = oracle.assign(X, C, msr, prior)
    if msr == 5:
        assert np.allclose(cost, ocost, rtol=2e-5, atol=1e-7)
        D = mc.cmp(X, C, msr=msr, prior=prior).astype(np.float64)
        got, best = D[np.arange(n), asn], D.min(1)
        assert np.allclose(got, best, rtol=0, atol=0)
        assert np.all((asn == oasn) | (np.abs(D[np.arange(n), oasn] - best) <= 4e-5 * np.abs(best) + 1e-7))
    else:
        assert np.array_equal(asn, oasn)
        assert np.array_equal(cost, ocost, equal_nan=True)


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_unaligned_device_rows(offset):
    """Rows that start 4 or 8 bytes past a 16-byte boundary (device views) take narrower copies."""
    import torch
    import minicore_gb300 as mc
    import oracle
    n, d, k = 333, 36, 21
    g = torch.Generator().manual_seed(3)
    buf = torch.randn(n * d + 8, generator=g)
    X = buf.cuda()[offset:offset + n * d].view(n, d)
    C = torch.randn(k, d, generator=g).numpy()
    job = mc.Job(X, C, msr=2)
    job.assign()
    asn, cost = np.empty(n, np.uint32), np.empty(n, np.float64)
    job.read(None, asn, cost)
    job.close()
    oasn, ocost = oracle.assign(buf[offset:offset + n * d].view(n, d).numpy(), C, 2, 0.0)
    assert np.array_equal(asn, oasn) and np.array_equal(cost, ocost)

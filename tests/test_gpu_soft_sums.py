"""Soft clustering's center sums add products rounded to float: the centers of one iteration over one and
two chunks of rows equal the rounded quotients of exact sums of those products."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(200, 2), (256, 5), (300, 33)])
def test_centers_are_sums_of_rounded_products(n, k):
    import minicore_gb300 as mc
    rng = np.random.default_rng(n)
    d = 150
    X = (1e4 + rng.standard_normal((n, d))).astype(np.float32)  # a product's rounding reaches the center's last bit
    r = mc.scluster(X, X[:k].copy(), msr=2, temp=0.05, maxiter=1)
    P = r["asn"]
    want = np.empty((k, d), np.float32)
    for c in range(k):
        den = math.fsum(P[:, c].tolist())
        for j in range(d):
            want[c, j] = math.fsum((P[:, c] * X[:, j]).tolist()) * (1.0 / den)
    assert np.array_equal(r["centers"], want)

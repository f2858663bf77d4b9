"""CSR k-means++ over wide matrices, at the column counts where the rounds change form: the center's row
beside the column loop (16,384 columns), in shared memory (28,672), read by the preparation itself
(1,572,864), with prior 1 and with prior 0, where every pair has a pv of its own.

The distances are compared with 64-bit sums over all columns of the terms of the float transforms.
Bound, with T the sum of the terms' parts (a |log a| + a |log b| for MKL, and so on): a float sum by 32
lanes is off by at most (d / 32 + 8) 2^-24 T, each logarithm, root or product by 2^-22 of its part."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
F = np.float32


def _side(pv, total, d):
    s = F(total + float(F(pv * F(d))))
    rsi = F(1) / s
    return rsi, F(pv * rsi)


def _distance(c, x, msr, prior):
    """The measure's sum for center row c and row x, and the bound of its error."""
    d = c.size
    sc, sx = float(c.sum(dtype=np.float64)), float(x.sum(dtype=np.float64))
    psum = prior * d
    least = F(F(7.0069e-42) * F(F(sc + psum) + F(sx + psum)))
    pv = least if F(prior) < least else F(prior)
    if msr in (0, 2):
        a, b = (c, x) if msr == 2 else (c + pv, x + pv)
        t = np.abs(a.astype(np.float64) - b)
        v, T = (t.sum(), t.sum()) if msr == 0 else ((t * t).sum(), ((np.abs(a) + np.abs(b)).astype(np.float64) ** 2).sum())
    else:
        (rc, ic), (rx, ix) = _side(pv, sc, d), _side(pv, sx, d)
        a, b = (c * rc + ic).astype(np.float64), (x * rx + ix).astype(np.float64)
        if msr == 6:
            v, T = ((np.sqrt(a) - np.sqrt(b)) ** 2).sum(), (a + b + 2 * np.sqrt(a * b)).sum()
        elif msr == 5:
            v, T = (a * (np.log(a) - np.log(b))).sum(), (a * (np.abs(np.log(a)) + np.abs(np.log(b)))).sum()
        else:
            m = a + b
            parts = [a * np.log(a), b * np.log(b), m * np.log(m / 2)]
            v, T = 0.5 * (parts[0] + parts[1] - parts[2]).sum(), 0.5 * sum(np.abs(p) for p in parts).sum()
    return max(v, 0.0), ((d / 32 + 8) * 2.0 ** -24 + 2.0 ** -22) * T


@pytest.mark.parametrize("msr,prior", [(0, 0.0), (2, 0.0), (4, 0.0), (4, 1.0), (5, 0.0), (5, 1.0), (6, 0.0), (6, 1.0)])
@pytest.mark.parametrize("n,d", [(45, 16384), (45, 16385), (70, 28672), (70, 28673), (33, 49153), (6, 1572864), (6, 1572865)])
def test_wide_rows(n, d, msr, prior):
    import minicore_gb300 as mc
    rng = np.random.default_rng(d + msr)
    rows = [np.sort(rng.choice(d, int(m), replace=False)) for m in rng.integers(40, 400, n)]
    ip = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    X = sp.csr_matrix((rng.random(ip[-1]).astype(F) * 4 + F(0.25), np.concatenate(rows).astype(np.int32), ip), shape=(n, d))
    k = 4
    ids, asn, costs = mc.kmeanspp(X, k, msr=msr, prior=prior, seed=9)
    assert len(set(ids.tolist())) == k
    D = np.asarray(X[ids].toarray(), F)
    for i in range(n):
        x = np.asarray(X[i].toarray(), F)[0]
        if i in ids:
            assert costs[i] == 0.0
            continue
        ref = [_distance(c, x, msr, prior) for c in D]
        got = costs[i] ** 2 * 2 if msr == 6 else costs[i]  # Hellinger: sqrt(v) / sqrt(2)
        slack = 2.0 ** -22 * got
        v, bound = ref[asn[i]]
        assert abs(got - v) <= bound + slack, (i, got, v, bound)
        for w, other in ref:  # the nearest, within the bounds
            assert v - bound <= w + other + slack


@pytest.mark.parametrize("msr", [0, 4, 5, 6])
@pytest.mark.parametrize("n,d", [(65535, 60), (65536, 60), (65600, 600)])
def test_many_rows_with_prior_zero(n, d, msr):
    """From 65,536 rows on the column loop with prior 0 is the kernel without shared memory: rows drawn from
    the whole range, the last one among them, have the bounded distances too."""
    import minicore_gb300 as mc
    rng = np.random.default_rng(d + msr)
    per = 9
    idx = np.sort(np.argsort(rng.random((n, 40)), axis=1)[:, :per] + rng.integers(0, d - 39, (n, 1)), axis=1)
    X = sp.csr_matrix((rng.random(n * per).astype(F) * 4 + F(0.25), idx.ravel().astype(np.int32),
                       np.arange(0, n * per + 1, per)), shape=(n, d))
    ids, asn, costs = mc.kmeanspp(X, 4, msr=msr, prior=0.0, seed=9)
    D = np.asarray(X[ids].toarray(), F)
    for i in [*rng.choice(n, 60).tolist(), n - 1]:
        if i in ids:
            assert costs[i] == 0.0
            continue
        ref = [_distance(c, np.asarray(X[i].toarray(), F)[0], msr, 0.0) for c in D]
        got = costs[i] ** 2 * 2 if msr == 6 else costs[i]
        slack = 2.0 ** -22 * got
        v, bound = ref[asn[i]]
        assert abs(got - v) <= bound + slack, (i, got, v, bound)
        for w, other in ref:
            assert v - bound <= w + other + slack

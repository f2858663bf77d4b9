"""Calls that run out of device memory: buffers that only make a call faster are given up, and a buffer
that did not fit is not asked for again.  (The allocations fail by a test hook; no memory is filled.)"""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _lib():
    from minicore_gb300 import _lib as m
    return m.load()


def _made():
    n = ctypes.c_uint64()
    _lib().mc_test_refuse_alloc(0, ctypes.byref(n))
    return n.value


def _counts(n, d, per, seed):
    rng = np.random.default_rng(seed)
    idx = np.concatenate([np.sort(rng.choice(d, per, replace=False)) for _ in range(n)]).astype(np.int32)
    return sp.csr_matrix((rng.integers(1, 5, n * per).astype(np.float32), idx, np.arange(0, n * per + 1, per)),
                         shape=(n, d))


@pytest.mark.parametrize("trials,lspp", [(1, 0), (3, 0), (1, 2)])
def test_seeding_gives_up_the_row_values(trials, lspp):
    """Once the entries' row sides are there, a later allocation that fails costs them, not the call."""
    import minicore_gb300 as mc
    X = _counts(500, 3000, 40, 1)
    kw = dict(msr=5, prior=1.0, seed=4, n_local_trials=trials, lspp=lspp)
    a0 = _made()
    want = mc.kmeanspp(X, 6, **kw)
    total = _made() - a0
    outcome = []
    for nth in range(1, total + 1):
        _lib().mc_test_refuse_alloc(nth, None)
        try:
            got = mc.kmeanspp(X, 6, **kw)
            for x, y in zip(want, got):
                assert np.array_equal(x, y)
            outcome.append(True)
        except MemoryError:
            outcome.append(False)
        finally:
            _lib().mc_test_refuse_alloc(0, None)
    first = outcome.index(True)  # the row values themselves, which may fail too
    assert first < total - 1 and not any(outcome[:first]) and all(outcome[first:])


def test_band_offsets_are_asked_for_once():
    import minicore_gb300 as mc
    X = _counts(2000, 4000, 300, 2)
    C = np.asarray(X[:10].toarray(), np.float32)

    def update(job):
        job.lloyd_step()
        out = np.empty((10, 4000), np.float32), np.empty(2000, np.uint32), np.empty(2000)
        job.read(*out)
        return out

    job = mc.Job(X, C, msr=5, prior=1.0)
    job.assign()
    a0 = _made()
    want = [update(job) for _ in range(3)]
    steps = _made() - a0
    job.close()
    gave_up = 0
    for nth in range(1, steps + 1):
        job = mc.Job(X, C, msr=5, prior=1.0)
        job.assign()
        _lib().mc_test_refuse_alloc(nth, None)
        try:
            got = [update(job)]
        except MemoryError:
            job.close()
            continue
        finally:
            _lib().mc_test_refuse_alloc(0, None)
        a0 = _made()
        got += [update(job) for _ in range(2)]
        assert _made() == a0  # nothing is tried again
        job.close()
        gave_up += 1
        for x, y in zip(want, got):
            assert all(np.array_equal(p, q) for p, q in zip(x, y))
    assert gave_up == 1


def test_jsd_logarithms_are_asked_for_once():
    import minicore_gb300 as mc
    n, d, k = 900, 3000, 40
    X = _counts(n, d, 200, 3)
    X.data[:] = 1.0  # one row sum: 30 x 120,000 entries take a table of a few groups
    for i in range(n):
        X.data[X.indptr[i]:X.indptr[i] + i % 30] = 2.0
    C = np.asarray(X[:k].toarray(), np.float32) + np.float32(0.5)

    def assign(job):
        job.assign()
        out = np.empty(n, np.uint32), np.empty(n)
        job.read(None, *out)
        return out

    job = mc.Job(X, C, msr=4, prior=1.0)
    a0 = _made()
    want = assign(job)
    total = _made() - a0
    job.close()
    gave_up = 0
    for nth in range(1, total + 1):
        job = mc.Job(X, C, msr=4, prior=1.0)
        _lib().mc_test_refuse_alloc(nth, None)
        try:
            got = [assign(job)]
        except MemoryError:
            job.close()
            continue
        finally:
            _lib().mc_test_refuse_alloc(0, None)
        a0 = _made()
        got.append(assign(job))
        assert _made() == a0
        job.close()
        gave_up += 1
        for g in got:
            assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1])
    assert gave_up == 1

"""Alias table over probabilities with infinities: a finite one's share of the infinite total is 0 and
its alias the last infinite point; every infinite point keeps its own slot."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,where", [(2, [1]), (7, [2, 5]), (300, [0, 1, 299]), (5000, [17, 18, 19, 4000]), (3, [0, 1, 2])])
def test_infinite_probabilities(n, where):
    import minicore_gb300 as mc
    from minicore_gb300 import _lib
    lib = _lib.load()
    probs = np.random.default_rng(n).random(n).astype(np.float32)
    probs[where] = np.inf
    h = ctypes.c_void_p()
    _lib.check(lib.mc_sampler_from_probs(mc.default_context().handle, n, mc._p(probs), None, ctypes.byref(h)))
    prob, alias = np.empty(n, np.float64), np.empty(n, np.uint32)
    _lib.check(lib.mc_sampler_alias(h, mc._p(prob), mc._p(alias)))
    lib.mc_sampler_destroy(h)
    want_p, want_a = np.zeros(n), np.full(n, where[-1], np.uint32)
    want_p[where], want_a[where] = 1.0, where
    assert np.array_equal(prob, want_p)
    assert np.array_equal(alias, want_a)

"""k-means++ outputs converted on the device equal the wide outputs converted on the host."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nbytes", [(1, 1), (256, 1), (257, 2), (300, 4)])
@pytest.mark.parametrize("f32", [0, 1])
def test_narrow_outputs(k, nbytes, f32):
    import minicore_gb300 as mc
    from minicore_gb300 import _lib
    rng = np.random.default_rng(k)
    n, d = 1031, 20
    X = rng.normal(size=(n, d)).astype(np.float32)
    M = mc._MatrixArg(X)
    u = mc.uniforms(3, k)
    h = mc.default_context().handle
    ids, asn, cost = np.empty(k, np.uint32), np.empty(n, np.uint32), np.empty(n, np.float64)
    _lib.check(_lib.load().mc_kmeanspp(h, M.ref, k, 2, 0.0, None, mc._p(u), mc._p(ids), mc._p(asn), mc._p(cost)))
    ids2 = np.empty(k, np.uint32)
    asn2 = np.empty(n, {1: np.uint8, 2: np.uint16, 4: np.uint32}[nbytes])
    cost2 = np.empty(n, np.float32 if f32 else np.float64)
    _lib.check(_lib.load().mc_kmeanspp_narrow(h, M.ref, k, 2, 0.0, None, mc._p(u), mc._p(ids2), mc._p(asn2), nbytes,
                                              mc._p(cost2), f32))
    assert np.array_equal(ids, ids2)
    assert np.array_equal(asn.astype(asn2.dtype), asn2)
    assert np.array_equal(cost.astype(cost2.dtype), cost2)


def test_narrow_refuses_a_type_too_small():
    import minicore_gb300 as mc
    from minicore_gb300 import _lib
    X = np.zeros((300, 2), np.float32)
    M = mc._MatrixArg(X)
    buf = np.empty(4096, np.uint8)
    p = buf.ctypes.data_as(ctypes.c_void_p)
    u = mc.uniforms(3, 257)
    for nbytes in (1, 3):
        with pytest.raises(ValueError):
            _lib.check(_lib.load().mc_kmeanspp_narrow(mc.default_context().handle, M.ref, 257, 2, 0.0, None, mc._p(u), p, p,
                                                      nbytes, p, 0))

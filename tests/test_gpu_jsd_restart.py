"""Coreset minibatch over wide CSR count rows under JSD: the pass over all centers goes by row groups
(which stages 64 centers at a time), the pass over a few restarted centers, padded to 32, does not."""
import ctypes
import json

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def test_restart_passes_leave_the_row_groups():
    import minicore_gb300 as mc
    from minicore_gb300 import _lib
    L = _lib.load()
    rng = np.random.default_rng(5)
    d, k, copies = 2100, 50, 5
    rows = []
    for g in range(30):  # 30 row sums, 14 rows each: a sample of 100 has too few rows per group
        for _ in range(14):
            r = np.zeros(d, np.float32)
            r[rng.choice(d, 900 + g, replace=False)] = 1.0
            rows.append(r)
    D = np.stack(rows)[rng.permutation(420)]
    X = sp.csr_matrix(D)
    X.sort_indices()
    # copies of center 0 win no row: restarted at every check-in they are empty at
    C0 = np.concatenate([D[:k - copies], np.repeat(D[:1], copies, 0)])
    L.mc_profile_reset()
    L.mc_profile_enable(1)
    try:
        res = mc.hcluster(X, C0, msr=4, prior=1.0, mbsize=100, maxiter=4, ncheckins=2, reseed_count=0, seed=3, cs=True)
        buf = ctypes.create_string_buffer(1 << 16)
        _lib.check(L.mc_profile_report(buf, ctypes.c_uint64(len(buf))))
    finally:
        L.mc_profile_enable(0)
    phases = json.loads(buf.value.decode())
    assert phases["assign_jsd_groups"]["count"] == res["numiter"]  # one pass over all centers a round
    assert phases["assign_csr_sparse"]["count"] > phases["assign_jsd_groups"]["count"]
    assert np.isfinite(res["finalcost"]) and res["finalcost"] <= res["initcost"]

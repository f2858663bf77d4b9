"""Autotuner decisions recorded for the k-means++ rounds before they kept block sums are not applied to
today's: the families are timed again under keys of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,n,d", [("kmpp_run", 3000, 20), ("kmpp_prune", 140000, 64)])
def test_old_decisions_are_not_taken(family, n, d, tmp_path):
    import minicore_gb300 as mc
    X = np.random.default_rng(1).normal(size=(n, d)).astype(np.float32)
    mc.autotune(True)
    try:
        mc.autotune_reset()
        mc.kmeanspp(X, 5, msr=2, seed=3)
        key, = [k for k in mc.autotune_report()["entries"] if k.startswith(family + "|")]
        parts = key.split("|")
        old = "|".join(p for p in parts if p != "blk")
        assert old != key
        path = tmp_path / "old.tsv"
        path.write_text(f"{old}\t1\t\n")
        mc.autotune_reset()
        mc.autotune_load(str(path))
        mc.kmeanspp(X, 5, msr=2, seed=3)
        got = mc.autotune_report()["entries"]
        assert key in got and len(got[key]["ms"]) >= 2  # timed anew
    finally:
        mc.autotune_reset()

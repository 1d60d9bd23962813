"""Batches past the sizes where their launches change: a scene whose SpMV has more
groups than its block cap takes at once (148 x 4 blocks of 256 groups of 4 cells, 606,208
cells), and more scenes than one launch of the layout kernels holds (16).  Every scene
comes out as a single call of it does, bit for bit."""
import numpy as np
import pytest

from test_batch import _batch_inputs, _single
from xfluid_b200 import scenes
from xfluid_b200.batch import BatchProjector

pytestmark = pytest.mark.gpu


def _equal_to_single(scs, precision, dtype):
    items = _batch_inputs(scs, dtype)
    bp = BatchProjector(precision, tol=1e-6, max_iter=400)
    try:
        assert bp.project(items)
        stats = bp.stats
    finally:
        bp.close()
    for q, (sc, it, st) in enumerate(zip(scs, items, stats)):
        rc, p, u, v, w, s1 = _single(sc, precision, dtype, 0)
        assert rc == 0 and st["status"] == 0 and st["graph"] == 1 and s1["graph"] == 1
        assert st["iterations"] == s1["iterations"], q
        for a, b in ((it["pressure"], p), (it["u"], u), (it["v"], v), (it["w"], w)):
            assert np.array_equal(a, b), q
    return stats


@pytest.mark.parametrize("precision,dtype", [("f64", np.float64), ("mixed", np.float32)])
def test_large_scene(precision, dtype):
    sc = scenes.blob_scene(dims=(96, 96, 96), seed=2, fractional=False, dtype=dtype)
    sc.mat[:] = scenes.FLUID
    sc.mat[-1] = scenes.AIR
    stats = _equal_to_single([sc, scenes.dam_break(24, seed=3, noise=0.3).astype(dtype)], precision, dtype)
    assert stats[0]["stored"] > 606208


def test_more_scenes_than_a_layout_launch():
    scs = [scenes.blob_scene(dims=(9 + q % 7, 8 + q % 5, 7 + q), seed=q, dtype=np.float64) for q in range(33)]
    _equal_to_single(scs, "f64", np.float64)

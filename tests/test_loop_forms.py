"""The PCG loop as a graph of any check_every and launched directly: the same bits."""
import numpy as np
import pytest

from gpu_util import make_ctx, project
from xfluid_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed", "f32"])
def test_forms_of_the_loop_agree(precision, monkeypatch):
    sc = scenes.blob_scene(dims=(37, 40, 33), seed=5, dtype=np.float64)
    out = {}
    for every in (0, 1, 2, 3, 5, 8, 25, 32, "direct"):
        if every == "direct":
            monkeypatch.setenv("XFP_KERNEL_EVENTS", "1")
        ctx = make_ctx(precision, tol=1e-5, max_iter=200, check_every=0 if every == "direct" else every)
        try:
            out[every] = project(ctx, sc)
        finally:
            ctx.close()
        assert out[every][0] == 0 and out[every][5]["graph"] == (0 if every == "direct" else 1)
    for every, got in out.items():
        assert got[5]["iterations"] == out[8][5]["iterations"] and got[5]["residual"] == out[8][5]["residual"], every
        for a, b in zip(got[1:5], out[8][1:5]):
            assert np.array_equal(a, b), every


def test_a_capped_loop_reports_its_cap():
    sc = scenes.blob_scene(dims=(37, 40, 33), seed=5, dtype=np.float64)
    for cap in (1, 4, 5, 7):
        ctx = make_ctx("f64", tol=1e-14, max_iter=cap)
        try:
            st = project(ctx, sc)[5]
            assert st["status"] == 1 and st["iterations"] == cap
        finally:
            ctx.close()


def test_one_context_for_grids_of_one_and_of_many_clusters():
    """The loop's executable graph passes from plain to cooperative sweeps and back."""
    scs = [scenes.blob_scene(dims=d, seed=5, fractional=False, dtype=np.float64) for d in ((24, 20, 22), (40, 65, 40))]
    want = []
    for sc in scs:
        ctx = make_ctx("f64", tol=1e-8, max_iter=300)
        try:
            want.append(project(ctx, sc))
        finally:
            ctx.close()
    ctx = make_ctx("f64", tol=1e-8, max_iter=300)
    try:
        for q in (0, 1, 0, 1, 1, 0):
            got = project(ctx, scs[q])
            assert got[0] == 0 and got[5]["graph"] == 1 and got[5]["iterations"] == want[q][5]["iterations"]
            for a, b in zip(got[1:5], want[q][1:5]):
                assert np.array_equal(a, b)
    finally:
        ctx.close()

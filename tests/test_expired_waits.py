"""A wait that runs out in any sweep of a projection (xfluid_b200/csrc/xfp_wave.cu):
the factorisation, the loop's first solves, the solves of the loop's graph, or of its
direct launches.  The call reports it, and the context then projects as a fresh one
does, bit for bit.  20 x 190 x 190 has 36 clusters' lines, more than are resident in
FP64, so tiles that are never handed out are waited for too."""
import numpy as np
import pytest

from gpu_util import make_ctx, project
from xfluid_b200 import scenes
from xfluid_b200._lib import XFP_ERR_TIMEOUT, XfpError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("events", [None, "1"])
@pytest.mark.parametrize("precision,dims", [("f64", (48, 48, 48)), ("mixed", (33, 65, 40)), ("f64", (20, 190, 190))])
def test_every_sweep_reports_an_expired_wait(precision, dims, events, monkeypatch):
    if events:
        monkeypatch.setenv("XFP_KERNEL_EVENTS", events)
    sc = scenes.blob_scene(dims=dims, seed=4, fractional=False, dtype=np.float64)
    kw = dict(tol=1e-8, max_iter=500)
    fresh = make_ctx(precision, **kw)
    ctx = make_ctx(precision, timeout_ms=20.0, **kw)
    try:
        want = project(fresh, sc)
        assert want[0] == 0 and want[5]["graph"] == (0 if events else 1)
        for n in range(1, 7):   # factor, forward, backward, then the loop's forward, backward, forward
            for _ in range(n):
                assert ctx.lib.xfp_debug_expire_next_sweep(ctx.ptr) == 0
            with pytest.raises(XfpError) as err:
                project(ctx, sc)
            assert err.value.code == XFP_ERR_TIMEOUT, n
            assert f"op {(0, 1, 2, 1, 2, 1)[n - 1]}," in str(err.value), n
            got = project(ctx, sc)
            assert got[0] == 0 and got[5]["iterations"] == want[5]["iterations"], n
            for a, b in zip(got[1:5], want[1:5]):
                assert np.array_equal(a, b), n
    finally:
        ctx.close()
        fresh.close()

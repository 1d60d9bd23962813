"""The extrapolation's layers as bits (xfluid_b200/csrc/xfp_steps.cu), 32 faces to
a word: rows around a word's length, layers that meet, end early or fill the
grid.  FP64 bit for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_util import make_ctx
from xfluid_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(30, 5, 4), (31, 4, 6), (32, 7, 3), (33, 3, 5), (63, 4, 4), (65, 9, 2), (2, 2, 2)])
@pytest.mark.parametrize("fill,layers", [(0.02, 1), (0.02, 4), (0.3, 12), (0.0, 2)])
def test_extrapolation_matches_the_oracle(dims, fill, layers):
    ni, nj, nk = dims
    rng = np.random.default_rng(ni + layers)
    mat = np.where(rng.random((nk, nj, ni)) < fill, scenes.FLUID, scenes.AIR).astype(np.uint8)
    sc = scenes.Scene(ni, nj, nk, mat, *[rng.standard_normal(s) for s in scenes.face_shapes(ni, nj, nk)])
    want = oracle.Oracle().extrapolate(sc, layers)
    got = [np.array(a) for a in (sc.u, sc.v, sc.w)]
    ctx = make_ctx("f64")
    try:
        ctx.check(ctx.lib.xfp_extrapolate_f64(ctx.ptr, ni, nj, nk, C.c_void_p(mat.ctypes.data),
                                              *(C.c_void_p(a.ctypes.data) for a in got), layers))
    finally:
        ctx.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)

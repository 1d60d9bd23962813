"""The wavefront sweeps (xfluid_b200/csrc/xfp_wave.cu) at the edges of their
decomposition: blocks of 8x8 lines, groups of 4 steps, clusters of 32x32 lines,
and more clusters' worth of lines than the chip holds at once."""
import numpy as np
import pytest

from gpu_util import bits_equal, debug_stages, make_ctx
from xfluid_b200 import scenes

pytestmark = pytest.mark.gpu

# ni, nj, nk: a block, its remainders, a second block / cluster by one line,
# lines shorter than a group, long lines, and 36 clusters' lines (FP64: 18 resident)
DIMS = [(8, 8, 8), (7, 9, 17), (3, 33, 32), (40, 65, 31), (300, 9, 9), (2, 34, 67), (20, 190, 190)]


def _scene(dims, kind):
    sc = scenes.blob_scene(dims=dims, seed=sum(dims), fractional=False, dtype=np.float64)
    if kind == "full":
        sc.mat[:] = scenes.FLUID
        sc.mat[-1] = scenes.AIR
    elif kind == "sparse":   # lone cells, so that most blocks and neighbours are empty
        m = np.random.default_rng(3).random(sc.mat.shape)
        sc.mat[:] = np.where(m < 0.004, scenes.FLUID, scenes.AIR)
        sc.mat.ravel()[sc.mat.size // 2] = scenes.FLUID
    return sc


@pytest.mark.parametrize("kind", ["full", "sparse"])
@pytest.mark.parametrize("dims", DIMS)
def test_stages(oracle_lib, dims, kind):
    """FP64: the factor and M^-1 r bit for bit.  Mixed: M^-1 is a sum over the
    grid's paths of non-negative products, at most ni+nj+nk factors long for
    each solve, and every factor carries at most 7 roundings (stored entry and
    pivot, product, three subtractions, scaling), so
    |dz| <= 14 (ni+nj+nk) 2^-24 M^-1 |r|, here with 1 % for the second order."""
    sc = _scene(dims, kind)
    A = oracle_lib.assemble(sc)
    F = oracle_lib.factor(sc, A)
    r = np.random.default_rng(2).standard_normal(A["diag"].shape).astype(np.float32).astype(np.float64) * (A["diag"] != 0)
    z = oracle_lib.precond(sc, F, r)
    ctx = make_ctx("f64")
    try:
        d = debug_stages(ctx, sc, r=r)
    finally:
        ctx.close()
    for k in ("inv", "lx", "ly", "lz"):
        assert bits_equal(d[k], F[k]), k
    assert bits_equal(d["z"], z)
    ctx = make_ctx("mixed")
    try:
        d = debug_stages(ctx, sc, r=r)
    finally:
        ctx.close()
    assert bits_equal(d["inv"], F["inv"])
    bound = 1.01 * 14 * sum(dims) * 2.0 ** -24 * oracle_lib.precond(sc, F, np.abs(r))
    assert np.all(np.abs(d["z"] - z) <= bound)

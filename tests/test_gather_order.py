"""The particle gathers (xfluid_b200/csrc/xfp_particles.cu) bit for bit against
a scan in the documented order: an output adds its particles by the bin of their
boxes' low corners (z, y, x), then by index."""
import numpy as np
import pytest

from gpu_util import make_ctx
from test_particles import _gpu_field, _gpu_p2g

pytestmark = pytest.mark.gpu


def _gather(P, ext, s, r, sh, dx, vcomp):
    unit = dx / s
    r2 = r * r
    c0, c1, c2 = (4.0 / 9.0) * (1.0 / (r2 * r2 * r2)), (17.0 / 9.0) * (1.0 / (r2 * r2)), (22.0 / 9.0) * (1.0 / r2)
    pos = P[:, :3] + sh
    lo, hi = np.trunc((-r + pos) / dx).astype(int), np.trunc((pos + r) / dx).astype(int)
    if s > 1:
        lo, hi = lo * s, (hi + 1) * s
    nb = (ext + s - 1) // s
    hits = np.all((hi >= 0) & (lo <= ext - 1), axis=1)
    b = np.minimum(np.maximum(lo, 0) // s, nb - 1)
    w, vw = np.zeros(ext[::-1]), np.zeros(ext[::-1])
    for q in np.lexsort((np.arange(len(P)), b[:, 0], b[:, 1], b[:, 2])):
        if not hits[q]:
            continue
        a, e = np.maximum(lo[q], 0), np.minimum(hi[q], ext - 1)
        d = [pos[q, n] - (np.arange(a[n], e[n] + 1) + 0.5) * unit for n in range(3)]
        xx, yy, zz = d[0] * d[0], d[1] * d[1], d[2] * d[2]
        rs = (xx[None, None, :] + yy[None, :, None]) + zz[:, None, None]
        cw = np.where(rs < r2, ((1.0 - c0 * rs * rs * rs) + c1 * rs * rs) - c2 * rs, 0.0)
        at = tuple(slice(a[n], e[n] + 1) for n in (2, 1, 0))
        w[at] += cw
        if vcomp >= 0:
            vw[at] += P[q, 3 + vcomp] * cw
    if vcomp < 0:
        return w
    with np.errstate(invalid="ignore"):
        return np.where(w > 0.0000001, vw / np.where(w > 0.0000001, w, 1.0), 0.0)


# a block of outputs (4 x 4 x 2) and its remainders; one bin with more particles
# than a queue (64) holds; velocities that are not finite; positions outside
@pytest.mark.parametrize("dims,n,crowd", [((4, 4, 2), 40, 0), ((5, 7, 3), 150, 100), ((13, 6, 9), 1200, 0),
                                          ((33, 2, 2), 300, 70)])
def test_gathers_are_the_ordered_sums(dims, n, crowd):
    rng = np.random.default_rng(n)
    dx = 0.1
    P = np.zeros((n, 6))
    P[:, :3] = rng.uniform(-0.1, 1.1, (n, 3)) * np.array(dims) * dx
    P[:crowd, :3] = (np.array(dims) // 2 + rng.uniform(0.1, 0.9, (crowd, 3))) * dx
    P[:, 3:] = rng.standard_normal((n, 3))
    P[5, 3], P[17, 4], P[33, 5] = np.inf, np.nan, -np.inf
    ctx = make_ctx("f64")
    try:
        got = _gpu_p2g(ctx, dims, dx, P)
        for a in range(3):
            sh = np.zeros(3)
            sh[a] = 0.5 * dx
            want = _gather(P, np.array(dims) + (np.arange(3) == a), 1, 1.5 * dx, sh, dx, a)
            assert np.array_equal(got[a], want, equal_nan=True), a
        for s, r in ((2, 0.93 * dx), (3, 1.7 * dx), (1, 0.4 * dx)):
            mat = np.zeros(dims[::-1], np.uint8)
            phi, _ = _gpu_field(ctx, mat, dx, s, r, 0.4, P)
            assert np.array_equal(phi, _gather(P, np.array(dims) * s + 1, s, r, np.zeros(3), dx, -1)), (s, r)
    finally:
        ctx.close()

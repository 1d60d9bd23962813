"""A closed context gives back all its device memory, whatever ran on it."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import make_ctx, project
from test_host_faces import _run
from test_particles import _gpu_field, _gpu_p2g
from xfluid_b200 import scenes

pytestmark = pytest.mark.gpu


def _particles():
    dims, dx = (64, 64, 64), 1.0 / 64
    P = np.random.default_rng(1).uniform(0.1, 0.9, (200000, 6))
    ctx = make_ctx("f64")
    try:
        _gpu_p2g(ctx, dims, dx, P)
        _gpu_field(ctx, np.zeros(dims, np.uint8), dx, 2, 0.93 * dx, 0.4, P)
    finally:
        ctx.close()


def _extrapolate():
    ni, nj, nk = 5, 600, 600
    mat = np.zeros((nk, nj, ni), np.uint8)
    mat[::9] = scenes.FLUID
    f = [np.zeros(s) for s in scenes.face_shapes(ni, nj, nk)]
    ctx = make_ctx("f64")
    try:
        ctx.check(ctx.lib.xfp_extrapolate_f64(ctx.ptr, ni, nj, nk, *(C.c_void_p(a.ctypes.data) for a in (mat, *f)), 2))
    finally:
        ctx.close()


def _project():
    ctx = make_ctx("mixed", tol=1e-6, max_iter=200)
    try:
        project(ctx, scenes.blob_scene(64, seed=7, dtype=np.float64))
    finally:
        ctx.close()


def _pinned_faces():
    _run(scenes.blob_scene(dims=(8, 600, 400), seed=7, dtype=np.float32), "pinned")


@pytest.mark.parametrize("work", [_project, _particles, _extrapolate, _pinned_faces])
def test_closed_contexts_hold_nothing(work):
    import torch
    work()   # (kernels are loaded, pinned pages cached)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(6):
        work()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    # (the driver maps memory by 2 MiB; every case held more than that in one context)
    assert before - torch.cuda.mem_get_info()[0] <= 2 << 20

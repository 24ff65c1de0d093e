"""Set-up work of vfs_poisson_lhs on the device: the count of connected fluid
regions (union-find) against a breadth-first search, and the coarsest level's
dense inverse (Gauss-Jordan by column blocks), the coarse masks (sandwich fill
in one block, or plane by plane on large levels)."""
from collections import deque

import numpy as np
import pytest

import oracle as O
from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _regions(fluid, per):
    """Regions of a [k, j, i] mask through faces; per = (i, j, k) periodic."""
    seen = np.zeros_like(fluid)
    n = 0
    for start in zip(*np.nonzero(fluid)):
        if seen[start]:
            continue
        n += 1
        seen[start] = True
        q = deque([start])
        while q:
            c = q.popleft()
            for ax in range(3):
                for s in (1, -1):
                    d = list(c)
                    d[ax] += s
                    m = fluid.shape[ax]
                    if not 0 <= d[ax] < m:
                        if not per[2 - ax]:
                            continue
                        d[ax] %= m
                    d = tuple(d)
                    if fluid[d] and not seen[d]:
                        seen[d] = True
                        q.append(d)
    return n


@pytest.mark.parametrize("per", [(1, 0, 1), (0, 0, 0), (1, 1, 1)])
@pytest.mark.parametrize("share", [0.25, 0.4, 0.9])  # below, near and above where the fluid joins up
def test_region_count(gpu_ctx, per, share):
    ni, nj, nk = 14, 9, 11
    rng = np.random.default_rng(91)
    nv = np.zeros((nk + 2, nj + 2, ni + 2))
    nv[1:-1, 1:-1, 1:-1] = np.where(rng.random((nk, nj, ni)) < share, 0.0, 4.0)
    g = synth.channel_case(ni, nj, nk, seed=92, levels=1).grid
    gid = gpu_ctx.grid_create(g.coor, nv, 1, 0, periodic=per)
    try:
        gpu_ctx.poisson_lhs(gid)
        assert gpu_ctx.grid_components(gid)[0] == _regions(nv[1:-1, 1:-1, 1:-1] < 0.1, per)
    finally:
        gpu_ctx.grid_destroy(gid)


@pytest.mark.parametrize("dims", [(3, 2, 3), (5, 4, 3), (10, 9, 7), (14, 12, 10), (16, 14, 15)])
def test_dense_inverse(gpu_ctx, dims):
    """One level: the preconditioner is the dense solve.  For a right-hand side
    of mean zero against the left null vector it returns A z = v; n eps times a
    condition number below 1e4 bounds the residual by 1e-8 at n = 3360 (there a
    block has half the columns)."""
    c = synth.channel_case(*dims, seed=93, levels=1)
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, 1, 0)
    try:
        gpu_ctx.poisson_lhs(gid)
        rng = np.random.default_rng(94)
        z0 = np.zeros(g.nvert.shape)
        z0[1:-1, 1:-1, 1:-1] = rng.normal(size=z0[1:-1, 1:-1, 1:-1].shape)
        v = gpu_ctx.apply_op(gid, 0, 1, z0)  # in the operator's range
        z = gpu_ctx.apply_precond(gid, capi.VFS_FP64, capi.default_params(precision="fp64"), v)
        r = gpu_ctx.apply_op(gid, 0, 1, z) - v
        assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(v)
    finally:
        gpu_ctx.grid_destroy(gid)


@pytest.mark.parametrize("dims,levels", [((16, 24, 16), 3), ((128, 112, 128), 2)])
def test_coarse_masks(gpu_ctx, dims, levels):
    """Blocks of solid cells at random, so that many coarse cells lie between
    solid ones on every axis: the masks are the oracle's."""
    ni, nj, nk = dims
    c = synth.channel_case(ni, nj, nk, seed=95, levels=levels)
    g = c.grid
    nv = np.zeros(g.nvert.shape)
    solid = np.random.default_rng(96).random((nk // 2, nj // 2, ni // 2)) < 0.5
    nv[1:-1, 1:-1, 1:-1] = solid.repeat(2, 0).repeat(2, 1).repeat(2, 2)
    gid = gpu_ctx.grid_create(g.coor, nv, levels, 1)
    mg = O.MG(O.dims_of(g), g.coor, nv, levels)
    try:
        for l in range(levels - 1):
            ref = mg.level_array(l, "nvert")
            assert np.array_equal(gpu_ctx.level_nvert(gid, l).ravel(), ref)
        assert ref.sum() > solid.sum()  # filled cells
    finally:
        mg.close()
        gpu_ctx.grid_destroy(gid)

"""The small levels of a V-cycle as one cluster launch against one launch per
operation.

The cluster launch uses the same device arithmetic in the same order, so one
V-cycle must agree bit for bit with the per-operation launches, which a
probed application runs.  The grids put the block split (k planes over 16 or
8 blocks) at its edges: fewer planes than blocks, a last block with fewer
planes, one plane, several planes a block; rows of odd pitch, a coarsest
order that is no multiple of a vector, bodies, and every combination of
periodic axes that reaches the halo planes' wrap."""
import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu

CASES = {
    # name: (ni, nj, nk, levels, periodic, spheres)
    "all_levels_small": (8, 6, 6, 2, (1, 0, 1), ()),
    "fewer_planes_than_blocks": (24, 20, 12, 3, (1, 0, 1), ()),
    "partial_last_block": (20, 8, 36, 3, (1, 0, 1), ()),
    "odd_coarsest": (52, 20, 36, 3, (1, 0, 1), [(3.0, 0.1, 1.5, 0.5)]),
    "finest_above": (104, 40, 72, 4, (1, 0, 1), [(3.0, 0.0, 1.5, 0.4)]),
    "channel_32": (32, 32, 32, 4, (1, 0, 1), ()),
    "large_top": (64, 32, 32, 3, (1, 0, 1), [(3.0, 0.0, 1.5, 0.6)]),
    "closed": (24, 16, 40, 3, (0, 0, 0), ()),
    "periodic_i_j": (24, 16, 40, 3, (1, 1, 0), ()),
    "periodic_k": (24, 16, 34, 2, (0, 0, 1), ()),
    "long_lines": (16, 128, 16, 3, (1, 0, 1), ()),
}


@pytest.mark.parametrize("sweeps", [(3, 3, -1, -1), (1, 2, 4, 1)])
@pytest.mark.parametrize("name", list(CASES))
def test_cluster_equals_separate_launches(gpu_ctx, name, sweeps):
    ni, nj, nk, levels, per, sph = CASES[name]
    c = synth.channel_case(ni, nj, nk, seed=51, beta=2.2, spheres=sph, levels=levels)
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, levels, c.immersed, periodic=per)
    try:
        gpu_ctx.poisson_lhs(gid)
        p = capi.default_params(nu1=sweeps[0], nu2=sweeps[1], nu1_coarse=sweeps[2], nu2_coarse=sweeps[3])
        v = np.random.default_rng(52).normal(size=g.nvert.shape)
        n0 = capi.launch_count()
        z = gpu_ctx.apply_precond(gid, capi.VFS_MIXED, p, v)
        fused = capi.launch_count() - n0
        gpu_ctx.probe_begin(capi.PROBE_ALL)
        try:
            n0 = capi.launch_count()
            zs = gpu_ctx.apply_precond(gid, capi.VFS_MIXED, p, v)
            separate = capi.launch_count() - n0
        finally:
            gpu_ctx.probe_end()
        assert fused < separate  # the cluster launch ran
        assert np.isfinite(z).all() and np.abs(z).max() > 0
        assert np.array_equal(z, zs), np.abs(z - zs).max()
    finally:
        gpu_ctx.grid_destroy(gid)

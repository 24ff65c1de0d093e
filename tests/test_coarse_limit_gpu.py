"""The largest level the cluster launch takes (32,768 cells: four cells a
thread on sixteen blocks) and the first one above it: launches of one V-cycle
and its result against the separate launches'."""
import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu

CASES = {
    # name: (dims, levels, launches): scale, then per level of its own three
    # pre-sweeps, restriction, prolongation and three post-sweeps, and the cluster
    "at": ((64, 64, 64), 4, 1 + 8 + 1),
    "above": ((72, 64, 64), 4, 1 + 16 + 1),  # 36 x 32 x 32 cells, then 18 x 16 x 16
}


@pytest.mark.parametrize("name", list(CASES))
def test_limit(gpu_ctx, name):
    dims, levels, launches = CASES[name]
    c = synth.channel_case(*dims, seed=55, levels=levels)
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, levels, 0)
    try:
        gpu_ctx.poisson_lhs(gid)
        p = capi.default_params()
        v = np.random.default_rng(56).normal(size=g.nvert.shape)
        n0 = capi.launch_count()
        z = gpu_ctx.apply_precond(gid, capi.VFS_MIXED, p, v)
        assert capi.launch_count() - n0 == launches
        gpu_ctx.probe_begin(capi.PROBE_ALL)
        try:
            zs = gpu_ctx.apply_precond(gid, capi.VFS_MIXED, p, v)
        finally:
            gpu_ctx.probe_end()
        assert np.isfinite(z).all() and np.abs(z).max() > 0
        assert np.array_equal(z, zs)
    finally:
        gpu_ctx.grid_destroy(gid)

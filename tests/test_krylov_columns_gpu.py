"""The Krylov reductions at the edges of their column chunks: the dots take up
to eight columns a sweep and the last block finishes them and closes the
Arnoldi column, so restart lengths below, at and past the chunk, on a grid of
one block and on one of several, must all reach the converged solution (the
parity bar of the pressure path: relative L2 of phi <= 1e-8 after removing
the fluid mean)."""
import numpy as np
import pytest

import oracle as O
from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu

GRIDS = {
    "one block": synth.channel_case(8, 6, 6, seed=41, levels=2),  # 640 cells with ghosts: two blocks at most
    "several blocks": synth.channel_case(24, 20, 12, seed=42, beta=2.8, levels=2),
}


@pytest.fixture(scope="module", params=list(GRIDS))
def solved(request):
    c = GRIDS[request.param]
    ref = O.projection_step(c.grid, c.ucont, levels=c.levels, immersed=0, rtol=1e-13, maxit=400)
    return c, ref


@pytest.mark.parametrize("orth", ["cgs", "cgs2"])
@pytest.mark.parametrize("restart", [3, 7, 8, 9, 17, 33])
def test_restart_lengths(gpu_ctx, solved, restart, orth):
    c, ref = solved
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, c.levels, c.immersed)
    try:
        gpu_ctx.poisson_lhs(gid)
        gpu_ctx.set_field(gid, capi.FIELD_USTAR, c.ucont)
        # one sweep a level: enough iterations to fill the longer cycles
        p = capi.default_params(rtol=1e-11, restart=restart, orth=orth, nu1=1, nu2=0, maxit=400)
        info, _ = gpu_ctx.projection_step(gid, p)
        phi = gpu_ctx.get_field(gid, capi.FIELD_PHI, g.nvert.shape)
        i = slice(1, -1)
        a, r = phi[i, i, i], ref["phi"].reshape(g.nvert.shape)[i, i, i]
        a, r = a - a.mean(), r - r.mean()
        assert info["converged"], info
        assert np.linalg.norm(a - r) <= 1e-8 * np.linalg.norm(r)
    finally:
        gpu_ctx.grid_destroy(gid)

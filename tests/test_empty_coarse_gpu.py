"""A mask whose coarsest level has no fluid row left, on a grid that had a
dense coarsest inverse before: a 2x2x2 fluid pocket in the solid is one fluid
cell of the next level, which the sandwich fill closes.  The step must equal
that of a grid created with this mask, in both precisions and in a batch, and
the grid must solve as before once the fluid is back."""
import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,grouped", [("mixed", 0), ("fp64", 0), ("mixed", 1)])
def test_coarsest_level_empties_and_fills(gpu_ctx, precision, grouped):
    c = synth.channel_case(16, 12, 16, seed=81, levels=2)
    open_nv = c.grid.nvert
    pocket = np.full_like(open_nv, 3.0)
    pocket[7:9, 5:7, 7:9] = 0.0  # fine cells 7, 8 of an axis are coarse cell 4, 5, 6 are 3
    ga = gpu_ctx.grid_create(c.grid.coor, open_nv, 2, 0)
    gb = gpu_ctx.grid_create(c.grid.coor, pocket, 2, 0)
    p = capi.default_params(precision=precision, rtol=1e-10, mg_grouped=grouped)

    def step(g):
        gpu_ctx.set_field(g, capi.FIELD_USTAR, c.ucont)
        gpu_ctx.set_field(g, capi.FIELD_P, np.zeros(open_nv.shape))
        infos, div = gpu_ctx.projection_step_batch([g], p)
        return infos[0]["iterations"], div[0], gpu_ctx.get_field(g, capi.FIELD_PHI, open_nv.shape)

    try:
        gpu_ctx.poisson_lhs(ga)
        first = step(ga)
        gpu_ctx.update_nvert(ga, pocket)
        gpu_ctx.poisson_lhs(ga)
        gpu_ctx.poisson_lhs(gb)
        assert not (gpu_ctx.level_nvert(ga, 0)[1:-1, 1:-1, 1:-1] < 0.1).any()
        a, b = step(ga), step(gb)
        assert a[:2] == b[:2] and np.array_equal(a[2], b[2])
        gpu_ctx.update_nvert(ga, open_nv)
        gpu_ctx.poisson_lhs(ga)
        again = step(ga)
        assert again[:2] == first[:2] and np.array_equal(again[2], first[2])
    finally:
        gpu_ctx.grid_destroy(ga)
        gpu_ctx.grid_destroy(gb)

"""The warp-row sweep on the general face form (terrain-following grids)
against the one-cell-per-thread gathers (explicit 32-column tiles, a multiple
of 8 columns on long lines): the same inputs and arithmetic per cell, so one
V-cycle must agree bit for bit.  A warp takes four rows at a time and 30
columns a tile: line lengths that leave 1, 2 or 3 rows over, a partial last
tile, bodies (one-sided cross terms), and periodic and closed axes; the
planes are enough for the sweep to be chosen (two blocks per SM)."""
import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu

CASES = {
    # name: (ni, nj, nk, levels, periodic, spheres)
    "rows_over_2": (64, 34, 104, 2, (1, 0, 1), [(3.1, 0.4, 1.5, 0.3)]),
    "rows_over_1_one_level": (40, 21, 160, 1, (1, 0, 1), ()),
    "rows_over_3_one_level": (62, 23, 110, 1, (0, 0, 0), [(3.1, 0.4, 1.5, 0.3)]),
    "periodic": (32, 32, 152, 2, (1, 1, 1), [(3.1, 0.4, 1.5, 0.3)]),
    "long_lines": (60, 256, 160, 3, (1, 0, 1), ()),
    # a sheared grid: the i and k faces have each other's cross term as well
    "sheared": (62, 23, 110, 1, (0, 0, 0), [(3.1, 0.4, 1.5, 0.3)]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_warp_rows_equal_single_cells(gpu_ctx, name):
    ni, nj, nk, levels, per, sph = CASES[name]
    coor = synth.terrain_coords(ni, nj, nk, 2.5)
    if name == "sheared":
        coor[: nk + 1, : nj + 1, : ni + 1, 0] += 0.3 * coor[: nk + 1, : nj + 1, : ni + 1, 2]
    nv = synth.sphere_nvert(coor, sph, *per) if sph else np.zeros((nk + 2, nj + 2, ni + 2))
    gid = gpu_ctx.grid_create(coor, nv, levels, 1 if sph else 0, periodic=per)
    try:
        gpu_ctx.poisson_lhs(gid)
        v = np.random.default_rng(83).normal(size=nv.shape)
        z = {c: gpu_ctx.apply_precond(gid, capi.VFS_MIXED, capi.default_params(smooth_cols=c), v) for c in (0, 32, 8)}
        assert np.isfinite(z[0]).all() and np.abs(z[0]).max() > 0
        assert np.array_equal(z[0], z[32]), np.abs(z[0] - z[32]).max()
        assert np.array_equal(z[0], z[8])
    finally:
        gpu_ctx.grid_destroy(gid)

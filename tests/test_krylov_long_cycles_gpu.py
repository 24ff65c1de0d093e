"""Krylov cycles that are filled to their last column: the dots take eight
columns a sweep, the iteration is replayed from a graph for any restart, and
64 columns is the longest cycle.  A strongly damped smoother makes the solve
take more iterations than the cycle has columns, which is asserted, so every
chunk and the restart after it run; the solution must reach the parity bar of
the pressure path (relative L2 of phi <= 1e-8 after removing the mean)."""
import numpy as np
import pytest

import oracle as O
from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu

# name: case, damping, restart lengths
GRIDS = {
    "two blocks": (synth.channel_case(8, 6, 6, seed=42, beta=2.8, levels=2), 0.2, (8, 9, 17, 33)),
    "several blocks": (synth.channel_case(24, 20, 12, seed=42, beta=2.8, levels=2), 0.05, (16, 17, 33, 64)),
    "more cells a thread": (synth.channel_case(48, 24, 32, seed=42, beta=2.8, levels=2), 0.2, (33, 64)),
}
RUNS = [(name, r) for name, g in GRIDS.items() for r in g[2]]


@pytest.fixture(scope="module")
def reference():
    kept = {}

    def of(name):
        if name not in kept:
            c = GRIDS[name][0]
            kept[name] = O.projection_step(c.grid, c.ucont, levels=c.levels, immersed=0, rtol=1e-13, maxit=400)["phi"]
        return kept[name]

    return of


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("orth", ["cgs", "cgs2"])
@pytest.mark.parametrize("name,restart", RUNS)
def test_filled_cycles(gpu_ctx, reference, name, restart, orth, precision):
    c, omega, _ = GRIDS[name]
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, c.levels, c.immersed)
    try:
        gpu_ctx.poisson_lhs(gid)
        gpu_ctx.set_field(gid, capi.FIELD_USTAR, c.ucont)
        p = capi.default_params(precision=precision, rtol=1e-11, restart=restart, orth=orth, nu1=1, nu2=0,
                                smoother="jacobi", omega=omega, maxit=800)
        info, _ = gpu_ctx.projection_step(gid, p)
        phi = gpu_ctx.get_field(gid, capi.FIELD_PHI, g.nvert.shape)
        assert info["converged"] and info["iterations"] > restart, info
        i = slice(1, -1)
        a, r = phi[i, i, i], reference(name).reshape(g.nvert.shape)[i, i, i]
        a, r = a - a.mean(), r - r.mean()
        assert np.linalg.norm(a - r) <= 1e-8 * np.linalg.norm(r)
    finally:
        gpu_ctx.grid_destroy(gid)

"""The FP64 sweep's line solve from both ends against the oracle's sweep (one
Thomas pass a line).  Line lengths around its cases: one or no row on a side of
the middle row, remainders of its four-row batches, even and odd lengths; tiles
of 32 columns (two warps a solve), 16 and 8; a body, whose identity rows cut a
line.  One sweep of damped line Jacobi: 1e-12 of the largest value bounds the
rounding of a solve of up to 64 rows (that grows with the square of the
length).  Long lines (tiles of 4 columns) by their backward error."""
import numpy as np
import pytest

import oracle as O
from vfs_v3p2_gb300 import synth

pytestmark = pytest.mark.gpu

CASES = {
    # name: (ni, nj, nk, spheres)
    "one_row_below": (6, 2, 5, ()),
    "one_row_each_side": (7, 3, 4, ()),
    "odd": (20, 9, 6, ()),
    "wide_tiles": (64, 10, 90, ()),
    "tiles_16": (36, 33, 80, [(3.1, 0.4, 1.5, 0.5)]),
    "tiles_8": (21, 64, 12, [(3.1, 0.4, 1.5, 0.5)]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_sweep_equals_oracle(gpu_ctx, name):
    ni, nj, nk, sph = CASES[name]
    c = synth.channel_case(ni, nj, nk, seed=101, levels=1, spheres=sph)
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, 1, 1 if sph else 0)
    mg = O.MG(O.dims_of(g), g.coor, g.nvert, 1)
    try:
        gpu_ctx.poisson_lhs(gid)
        rng = np.random.default_rng(102)
        b, x = rng.normal(size=(2,) + g.nvert.shape)
        for a in (b, x):
            a[g.nvert > 0.1] = 0.0
            a[0], a[-1], a[:, 0], a[:, -1], a[:, :, 0], a[:, :, -1] = 0, 0, 0, 0, 0, 0
        ref = x.copy()
        mg.smooth(0, b, ref, 1, 0.8)
        got = gpu_ctx.mg_smooth(gid, 0, b, x, 0.8)
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    finally:
        mg.close()
        gpu_ctx.grid_destroy(gid)


@pytest.mark.parametrize("dims", [(10, 400, 4), (12, 256, 8)])
def test_long_lines_backward_error(gpu_ctx, dims):
    """The correction solves a line system whose entries differ from T's by a few
    roundings: with |L| |U| <= 3 |T| (diagonal dominance) and nine roundings a
    row in factors and substitutions, 27 eps |T| |delta|, and 12 eps of the 11
    products of the residual; 32 eps of their sum bounds both, together with the
    rounding of the blend that delta is read back from."""
    c = synth.channel_case(*dims, seed=103, levels=1)
    g = c.grid
    gid = gpu_ctx.grid_create(g.coor, g.nvert, 1, 0)
    omega = 0.8
    try:
        gpu_ctx.poisson_lhs(gid)
        A = gpu_ctx.coef(gid, 0, 1).reshape((19,) + g.nvert.shape)
        b, x = np.random.default_rng(104).normal(size=(2,) + g.nvert.shape)
        for a in (b, x):
            a[0], a[-1], a[:, 0], a[:, -1], a[:, :, 0], a[:, :, -1] = 0, 0, 0, 0, 0, 0
        got = gpu_ctx.mg_smooth(gid, 0, b, x, omega)
        inner = (slice(None), slice(1, -1), slice(None))
        d = (got - x) / omega
        low, mid, high = A[4].copy(), A[0], A[3].copy()  # S, P, N
        low[:, 1], high[:, -2] = 0, 0
        line = lambda f, v: f(low[inner]) * v[:, :-2] + f(mid[inner]) * v[:, 1:-1] + f(high[inner]) * v[:, 2:]
        res = b - gpu_ctx.apply_op(gid, 0, 1, x)
        err = np.abs(line(lambda m: m, d) - res[inner])
        size = line(np.abs, np.abs(d) + 2 * (np.abs(x) + np.abs(got)) / omega) + np.abs(b)[inner]
        size += sum(np.abs(A[m]) for m in range(19))[inner] * np.abs(x).max()
        assert (err <= 32 * np.finfo(float).eps * size)[1:-1, :, 1:-1].all()
        assert np.abs(d).max() > 0.1
    finally:
        gpu_ctx.grid_destroy(gid)

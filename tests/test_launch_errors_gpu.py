"""A refused launch ends the solve with VFS_ERR_CUDA instead of leaving its
kernel out.  The line sweep has one row of blocks per k plane, so a grid of
more than 65535 planes asks for more than a launch may have and the runtime
refuses it on the host; other grids of the context solve as before."""
import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tall(gpu_ctx):
    c = synth.channel_case(4, 4, 66000, seed=91, levels=1)
    gid = gpu_ctx.grid_create(c.grid.coor, c.grid.nvert, 1, 0)
    gpu_ctx.poisson_lhs(gid)
    gpu_ctx.set_field(gid, capi.FIELD_USTAR, c.ucont)
    yield gid
    gpu_ctx.grid_destroy(gid)


def small_step(ctx):
    c = synth.channel_case(16, 12, 16, seed=92, levels=2)
    g = ctx.grid_create(c.grid.coor, c.grid.nvert, 2, 0)
    try:
        ctx.poisson_lhs(g)
        ctx.set_field(g, capi.FIELD_USTAR, c.ucont)
        return ctx.projection_step(g, capi.default_params(rtol=1e-10))[0]
    finally:
        ctx.grid_destroy(g)


@pytest.mark.parametrize("entry", ["step", "batch", "served", "precond"])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_refused_launch_is_reported(gpu_ctx, tall, precision, entry):
    before = small_step(gpu_ctx)
    p = capi.default_params(precision=precision, restart=4, maxit=8)
    if entry == "served":
        assert gpu_ctx.submit(tall, p) is not None
        _, status, _, _ = gpu_ctx.poll(wait=True)
        assert status == capi.VFS_ERR_CUDA
    else:
        with pytest.raises(capi.VfsError) as e:
            if entry == "step":
                gpu_ctx.projection_step(tall, p)
            elif entry == "precond":
                shape = (66002, 6, 6)
                gpu_ctx.apply_precond(tall, capi.VFS_MIXED if precision == "mixed" else capi.VFS_FP64, p, np.zeros(shape))
            else:
                gpu_ctx.projection_step_batch([tall], p)
        assert e.value.code == capi.VFS_ERR_CUDA and "refused" in str(e.value)
    after = small_step(gpu_ctx)
    assert before["converged"] and after["iterations"] == before["iterations"]

"""vfs_divergence_max_noalloc keeps nothing between calls: results of grids of
different sizes (one block to several per SM) called in turn, on two streams
at once with an output each, and replayed from a captured graph are those of
each call alone.  Outputs are poisoned before every call.  The expected value
is the same sequence of FP64 operations in numpy, so it is compared bit for
bit (a maximum does not depend on the block partition)."""
import ctypes

import numpy as np
import pytest

from vfs_v3p2_gb300 import capi

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (17, 9, 11), (66, 67, 68), (130, 66, 130)]


@pytest.fixture(scope="module")
def grids():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("torch has no CUDA device")
    dev = torch.device("cuda", 0)
    out = []
    for q, (mx, my, mz) in enumerate(SIZES):
        rng = np.random.default_rng(60 + q)
        u = rng.normal(size=(3, mz, my, mx))
        aj = 1.0 + rng.uniform(size=(mz, my, mx))
        i = slice(1, -1)
        div = (u[0, i, i, 1:-1] - u[0, i, i, :-2] + u[1, i, 1:-1, i] - u[1, i, :-2, i] + u[2, 1:-1, i, i] -
               u[2, :-2, i, i]) * aj[i, i, i]
        arrs = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (*u, aj, np.zeros((mz, my, mx)))]
        out.append(((mx, my, mz), arrs, float(np.abs(div).max())))
    torch.cuda.synchronize()
    return torch, dev, out


def call(grid, out_ptr, stream):
    (mx, my, mz), arrs, _ = grid
    err = ctypes.create_string_buffer(256)
    rc = capi.load().vfs_divergence_max_noalloc(0, mx, my, mz, 0, 0, 0, *[a.data_ptr() for a in arrs], out_ptr, stream,
                                                err, 256)
    assert rc == 0, err.value.decode()


def test_alternating_sizes(grids):
    torch, dev, gs = grids
    n = 4 * len(gs)
    out = torch.full((n,), 1e300, dtype=torch.float64, device=dev)
    s = torch.cuda.current_stream().cuda_stream
    for q in range(n):
        call(gs[q % len(gs)], out.data_ptr() + 8 * q, s)
    torch.cuda.synchronize()
    assert out.tolist() == [gs[q % len(gs)][2] for q in range(n)]


def test_overlapping_streams(grids):
    torch, dev, gs = grids
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    n = 64
    out = torch.full((2, n), -1.0, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    for q in range(n):
        for r, st in enumerate(streams):
            call(gs[2 + (q + r) % 2], out.data_ptr() + 8 * (r * n + q), st.cuda_stream)
    torch.cuda.synchronize()
    for r in range(2):
        assert out[r].tolist() == [gs[2 + (q + r) % 2][2] for q in range(n)]
    # and a call alone afterwards
    test_alternating_sizes(grids)


def test_captured(grids):
    torch, dev, gs = grids
    out = torch.full((len(gs),), -1.0, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream().cuda_stream
        for q, grid in enumerate(gs):
            call(grid, out.data_ptr() + 8 * q, s)
    for _ in range(3):
        out.fill_(7e200)
        g.replay()
        torch.cuda.synchronize()
        assert out.tolist() == [grid[2] for grid in gs]

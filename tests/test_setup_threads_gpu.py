"""Operators set up in two threads at once, each on a context of its own: the
dense coarsest inverse of a large order (512 panels) while small orders are
inverted beside it must be the one it is alone, bit for bit (the panels'
order of operations does not depend on what else runs)."""
import threading

import numpy as np
import pytest

from vfs_v3p2_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def test_dense_inverse_beside_smaller_ones():
    large = synth.channel_case(16, 16, 16, seed=71, beta=2.0, levels=1)  # order 4096
    small = synth.channel_case(8, 6, 6, seed=72, levels=1)  # order 288
    p = capi.default_params()
    v = np.random.default_rng(73).normal(size=large.grid.nvert.shape)
    with capi.Context(0) as a, capi.Context(0) as b:
        ga = a.grid_create(large.grid.coor, large.grid.nvert, 1, 0)
        gb = b.grid_create(small.grid.coor, small.grid.nvert, 1, 0)
        a.poisson_lhs(ga)
        alone = a.apply_precond(ga, capi.VFS_FP64, p, v)
        stop = threading.Event()
        turns, errors = [0], []

        def beside():
            try:
                while not stop.is_set():
                    b.poisson_lhs(gb)
                    turns[0] += 1
            except Exception as e:  # noqa: BLE001 (reported by the main thread)
                errors.append(e)

        t = threading.Thread(target=beside)
        t.start()
        try:
            for _ in range(5):
                a.poisson_lhs(ga)
                got = a.apply_precond(ga, capi.VFS_FP64, p, v)
                assert np.array_equal(got, alone)
        finally:
            stop.set()
            t.join()
        assert not errors and turns[0] > 0
        assert np.isfinite(alone).all() and np.abs(alone).max() > 0

"""The grid build orders slots by cell and, in a cell, by original index: worlds
of one cell and of many scan tiles, cells of one particle and of several hundred,
particle counts around a warp and a block, and a second build from the first
one's order."""
import numpy as np
import pytest

import physics_engine_rs as pe
from helpers import dam_break_params_pe

pytestmark = pytest.mark.gpu

H = 0.02  # the cells' side is 2 h


@pytest.mark.parametrize("n,extent,dim", [(1, 0.03, 3), (31, 0.03, 3), (700, 0.03, 3), (257, 2.0, 3), (6000, 0.4, 3),
                                          (3000, 6.0, 2), (5001, 0.5, 2)])
def test_order_is_by_cell_then_index(n, extent, dim):
    rng = np.random.default_rng(n)
    x = rng.uniform(0.0, extent, (n, 3))
    x[: n // 2] = x[: n // 2] ** 2 / extent  # crowded towards the origin
    if dim == 2:
        x[:, 2] = 0.0
    p = pe.Particles(dim, 1000.0, 1e-3, H)
    for a in x:
        p.push_fluid(tuple(a))
    w = pe.WcsphWorld(p, dam_break_params_pe(False))
    for _ in range(2):
        w.rebuild_grid()
        got = w.grid()
        keys = np.floor(x * (1.0 / (2.0 * H))).astype(np.int64)
        if dim == 2:
            keys[:, 2] = 0
        order = np.lexsort((np.arange(n), keys[:, 2], keys[:, 1], keys[:, 0]))
        cells, first, count = np.unique(keys[order], axis=0, return_index=True, return_counts=True)
        assert np.array_equal(got["order"], order)
        assert np.array_equal(got["keys"], keys)
        assert np.array_equal(got["occupied"], cells)
        assert np.array_equal(got["ranges"], np.stack([first, first + count], 1))
        x = x[rng.permutation(n)]
        w.set_positions(x)
    w.close()

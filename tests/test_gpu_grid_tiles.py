"""The grid's scan over domains of few and of many tiles (4,096 cells each): up to 1,536 tiles every tile adds up
the ones before it, beyond them one block scans their sums first, 4,096 of them at a time."""
import numpy as np
import pytest

import physics_engine_rs as pe
from helpers import assert_bits_equal, dam_break_params_pe

pytestmark = pytest.mark.gpu


def _world(margin):
    # particles near both ends of the domain, so that occupied cells lie in its first and last tiles
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(0.0, 0.1, (300, 3)), 6.0 + rng.uniform(0.0, 0.1, (400, 3)),
                        rng.uniform(0.0, 6.1, (50, 3))])
    p = pe.Particles(3, 1000.0, 1e-3, 0.02)
    for k, a in enumerate(x):
        p.push_boundary(tuple(a), 1e-6) if k % 5 == 4 else p.push_fluid(tuple(a))
    return pe.WcsphWorld(p, dam_break_params_pe(False), pe.WcsphConfig(domain_margin=0.0, domain_margin_cells=margin)), len(x)


@pytest.mark.parametrize("margin,tiles", [(15, (1, 1536)), (17, (1536, 4096)), (56, (4096, 8192)), (57, (4096, 8192))])
def test_the_scan_of_many_tiles(margin, tiles):
    w, n = _world(margin)
    ref, _ = _world(4)
    assert tiles[0] < -(-w.capacity_info()["dense_cells"] // 4096) <= tiles[1]
    for one in (w, ref):
        one.rebuild_grid()
    for _ in range(2):
        a, b = w.grid(), ref.grid()
        for k in ("order", "keys", "occupied", "ranges"):
            assert np.array_equal(a[k], b[k]), k
        assert len(a["order"]) == n
        for one in (w, ref):
            one.run(1e-6, 2)
        assert_bits_equal(w.positions(), ref.positions(), "x")
        assert_bits_equal(w.densities(), ref.densities(), "rho")
    w.close()
    ref.close()

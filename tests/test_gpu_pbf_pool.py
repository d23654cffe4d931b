"""The list pool of a PBF world whose parameters come to keep the cells through several constraint iterations:
sized again, by all candidates, where it was sized by those in support."""
import numpy as np
import pytest

import physics_engine_rs as pe
from helpers import assert_bits_equal

pytestmark = pytest.mark.gpu

DX = 0.02


def _world(iterations, reuse, neighbours):
    p = pe.Particles(3, 1000.0, pe.mass_from_spacing(1000.0, DX, 3), 2 * DX)
    p.fill_box((0.4, 0.4, 0.4), 14, 13, 12, DX)
    p.jitter_fluid(3, 0.05 * DX)
    p.fill_box_boundary((0.0, 0.0, 0.0), (1.2, 1.2, 1.2), 2 * DX, 1)
    prm = pe.PbfParams(iterations=iterations, reuse_neighbours=reuse, gravity=(0.0, 0.0, 0.0))
    return pe.PbfWorld(p, prm, pe.WcsphConfig(max_neighbours=neighbours))  # few: the first build sizes the pool


@pytest.mark.parametrize("iterations,reuse", [(1, True), (4, False)])
def test_a_pool_sized_in_support_grows_for_kept_cells(iterations, reuse):
    small, ample = _world(iterations, reuse, 4), _world(iterations, reuse, 8192)
    dt = 1e-3
    n = 14 * 13 * 12
    for w in (small, ample):
        w.run(dt, 1)
        p = w.params
        p.iterations, p.reuse_neighbours = 4, True
        w.params = p
        x = w.positions()
        v = np.zeros_like(x)
        v[:n] = (x[:n].mean(0) - x[:n]) * (0.5 / dt)  # predicted: an eighth of the volume
        w.set_velocities(v)
        w.run(dt, 1)
        assert w.status() & pe.STATUS_NEIGHBOUR_OVERFLOW == 0
    for a, b, what in ((small.positions(), ample.positions(), "x"), (small.velocities(), ample.velocities(), "v"),
                       (small.densities(), ample.densities(), "rho"), (small.lambdas(), ample.lambdas(), "lambda")):
        assert np.isfinite(a).all()
        assert_bits_equal(a, b, what)
    small.close()
    ample.close()

"""Positions set by the host without a rebuild of the grid: the reference still takes a particle's candidates
from the cells of the last grid, however far the positions have gone since, and decides by the present
distances. The lists of the f64 passes have to hold every pair in support."""
import numpy as np
import pytest

import oracle as O
import physics_engine_rs as pe
from helpers import assert_bits_equal, dam_break_params_pe

pytestmark = pytest.mark.gpu

CELL = 0.04  # 2 h


def _worlds(dim):
    mass = pe.mass_from_spacing(1000.0, 0.01, dim)
    scenes = []
    for S in (pe.Particles, O.Scene):
        s = S(dim, 1000.0, mass, 0.02)
        s.fill_box((0.02, 0.02, 0.02 if dim == 3 else 0.0), 11, 9, 8 if dim == 3 else 1, 0.01)
        s.fill_box_boundary((0.0, 0.0, 0.0), (0.2, 0.15, 0.14 if dim == 3 else 0.0), 0.01, 1)
        scenes.append(s)
    return (pe.WcsphWorld(scenes[0], dam_break_params_pe(False)),
            O.World(scenes[1], O.dam_break_params(materialize=False)), scenes[0].arrays())


def _follow(w, o, x, v):
    w.set_positions(x)
    o.set_x(x)
    w.set_velocities(v)
    o.set_v(v)
    for one in (w, o):
        one.compute_density()
        one.compute_pressure()
        one.compute_forces()
    assert_bits_equal(w.densities(), o.rho(), "rho")
    assert_bits_equal(w.accelerations(), o.a(), "a")
    assert_bits_equal(w.boundary_forces(), o.boundary_force(), "boundary force")
    for a, b in zip(w.neighbour_counts(), o.neighbour_counts()):
        np.testing.assert_array_equal(a.astype(np.int64), b)
    w.apply_xsph()
    o.apply_xsph()
    assert_bits_equal(w.velocities(), o.v(), "v")


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("cells", [0.0, 0.45, 0.7, 1.0, 5.0, 10.0, 100.0, 300.0, 1e5])
def test_every_particle_shifted(cells, dim):
    w, o, a = _worlds(dim)
    w.rebuild_grid()
    o.rebuild_grid()
    rng = np.random.default_rng(3)
    x = a["x"] + rng.uniform(-1e-3, 1e-3, a["x"].shape) + cells * CELL * np.array([0.6, -0.7, 0.4])
    v = rng.normal(0.0, 0.1, x.shape)
    if dim == 2:
        x[:, 2] = v[:, 2] = 0.0
    _follow(w, o, x, v)
    # and back: the lists are those of the cells again
    back = a["x"].copy()
    _follow(w, o, back, v)
    w.close()


@pytest.mark.parametrize("cells", [0.6, 3.0, 40.0, 2000.0])
def test_some_particles_shifted(cells):
    """A third of the fluid and a few boundary samples go, each into one of two directions: the unions hold
    near and far candidates, and the far ones have neighbours among themselves."""
    w, o, a = _worlds(3)
    w.rebuild_grid()
    o.rebuild_grid()
    rng = np.random.default_rng(4)
    x = a["x"] + rng.uniform(-1e-3, 1e-3, a["x"].shape)
    way = np.where(rng.random(len(x)) < 0.5, 1.0, -1.0)[:, None] * np.array([0.5, 0.8, -0.3])
    x = np.where((rng.random(len(x)) < 0.33)[:, None], x + cells * CELL * way, x)
    _follow(w, o, x, rng.normal(0.0, 0.1, x.shape))
    w.close()


def test_a_particle_beyond_single_precision_leaves_the_others_alone():
    w, o, a = _worlds(3)
    w.rebuild_grid()
    o.rebuild_grid()
    x = a["x"].copy()
    x[5] = (1e30, 0.05, 0.05)
    x[17] = (0.05, -1e42, 0.05)  # its offset is infinite in single precision
    _follow(w, o, x, np.zeros_like(x))
    w.close()

"""Every lane count of the f64 pair passes reproduces the oracle bit for bit:
lists of 0 to 17 entries (shorter than, equal to and just beyond a round of
any lane count, with rows of one to four entries), lists longer than the force
pass's queue, oriented and plain boundary samples, both viscosity terms, the
other kernels, 2-D, and XSPH with and without the kept weights."""
import numpy as np
import pytest

import oracle as O
import physics_engine_rs as pe
from helpers import assert_bits_equal, dam_break_params_pe

pytestmark = pytest.mark.gpu

DX = 0.01


def clusters(s):
    """Groups of 1, 2, ... 18 fluid particles out of each other's reach, some with boundary samples."""
    rng = np.random.default_rng(11)
    for k in range(1, 19):
        c = np.array([0.3 * (k % 5), 0.3 * (k // 5), 0.05])
        for _ in range(k):
            s.push_fluid(tuple(c + rng.uniform(-0.008, 0.008, 3)), tuple(rng.uniform(-0.5, 0.5, 3)))
        if k % 3 == 0:
            s.push_boundary(tuple(c + np.array([0.0, 0.0, -0.02])), DX**3)
        if k % 4 == 0:
            wall = (tuple(c + np.array([0.0, 0.02, 0.0])), DX**3, (0.0, -1.0, 0.0))
            s.push_boundary_oriented(*wall) if isinstance(s, pe.Particles) else s.push_boundary(*wall)


def dense(s):
    """A block at 0.62 of the spacing: ~1,000 neighbours in support for its inner particles."""
    s.fill_box((0.02, 0.02, 0.02), 11, 11, 11, 0.62 * DX)
    s.jitter_fluid(3, 1e-4)
    s.fill_box_boundary((0.0, 0.0, 0.0), (0.12, 0.12, 0.12), DX, 1)


def tank(s):
    s.fill_box((DX, DX, DX), 9, 7, 6, DX)
    s.jitter_fluid(5, 1e-4)
    s.fill_box_boundary((0.0, 0.0, 0.0), (0.2, 0.1, 0.12), DX, 1)


def planar(s):
    s.fill_box((DX, DX, 0.0), 13, 11, 1, DX)
    s.jitter_fluid(7, 1e-4)
    s.fill_box_boundary((0.0, 0.0, 0.0), (0.3, 0.2, 0.0), DX, 1)


SCENES = {
    "clusters": (clusters, 3, 0, 0.0, 6),
    "dense": (dense, 3, 0, 0.0, 2),
    "tank, beta, Wendland": (tank, 3, 1, 0.3, 6),
    "tank, poly6": (tank, 3, 2, 0.0, 4),
    "planar": (planar, 2, 0, 0.0, 6),
}


@pytest.mark.parametrize("scene", list(SCENES))
def test_lane_counts_bit_exact(scene):
    build, dim, kernel, beta, steps = SCENES[scene]
    mass = pe.mass_from_spacing(1000.0, DX, dim)
    ps, os_ = pe.Particles(dim, 1000.0, mass, 2 * DX), O.Scene(dim, 1000.0, mass, 2 * DX)
    build(ps)
    build(os_)
    op = O.dam_break_params(materialize=False)
    op.kernel, op.visc_beta = kernel, beta
    o = O.World(os_, op)
    dt = 1e-5
    o.run(dt, steps)
    for lanes in (0, 1, 4, 8, 16, 32):
        for weights in (True, False):
            prm = dam_break_params_pe(False)
            prm.density_kernel, prm.visc_beta = kernel, beta
            w = pe.WcsphWorld(ps, prm)
            w.set_lanes(lanes)
            w.set_pair_weights(weights)
            w.run(dt, steps)
            what = f"{scene}, {lanes} lanes, weights {weights}"
            assert_bits_equal(w.positions(), o.x(), what + " x")
            assert_bits_equal(w.velocities(), o.v(), what + " v")
            assert_bits_equal(w.densities(), o.rho(), what + " rho")
            assert_bits_equal(w.accelerations(), o.a(), what + " a")
            assert_bits_equal(w.boundary_forces(), o.boundary_force(), what + " boundary force")
            if scene == "dense" and lanes == 1:
                assert int(w.neighbour_counts()[1].max()) > 512
            w.close()


def test_unknown_lane_counts_are_refused():
    ps = pe.Particles(3, 1000.0, pe.mass_from_spacing(1000.0, DX, 3), 2 * DX)
    tank(ps)
    w = pe.WcsphWorld(ps, dam_break_params_pe(False))
    for lanes in (2, 3, 64):
        with pytest.raises(pe.PeError):
            w.set_lanes(lanes)
    w.close()

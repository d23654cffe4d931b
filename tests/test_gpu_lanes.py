"""Every lane count of the pair passes reproduces the oracle bit for bit (single
precision: the one-lane form):
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


@pytest.mark.parametrize("scene", list(SCENES)[:3] + ["planar"])
def test_single_precision_lane_counts_agree(scene):
    """The compensated sums of the single-precision form come out the same bits for 1, 8 and 32 lanes."""
    build, dim, _, beta, steps = SCENES[scene]
    ps = pe.Particles(dim, 1000.0, pe.mass_from_spacing(1000.0, DX, dim), 2 * DX)
    build(ps)
    prm = dam_break_params_pe(False)
    prm.visc_beta, prm.precision = beta, pe.PRECISION_F32
    for weights in (True, False):
        want = None
        for lanes in (1, 8, 32, 0):
            w = pe.WcsphWorld(ps, prm)
            w.set_lanes(lanes)
            w.set_pair_weights(weights)
            w.run(1e-5, steps)
            got = [w.positions(), w.velocities(), w.densities(), w.accelerations()]
            w.close()
            want = want or got
            for a, b, what in zip(got, want, ("x", "v", "rho", "a")):
                assert_bits_equal(a, b, f"{scene}, {lanes} lanes, weights {weights} {what}")


def test_unknown_lane_counts_are_refused():
    ps = pe.Particles(3, 1000.0, pe.mass_from_spacing(1000.0, DX, 3), 2 * DX)
    tank(ps)
    w = pe.WcsphWorld(ps, dam_break_params_pe(False))
    for lanes in (2, 3, 64):
        with pytest.raises(pe.PeError):
            w.set_lanes(lanes)
    w.close()


@pytest.mark.parametrize("dim,kernel", [(3, 0), (3, 1), (2, 0)])
def test_dfsph_lane_counts_bit_exact(dim, kernel):
    """The divergence-free solver's pair passes with 1, 8 and 32 lanes: plates of oriented samples, warm start,
    boundary reactions, lists whose lengths are no multiple of any lane count."""
    dx = 0.05
    mass = pe.mass_calibrated_to_rest(1000.0, dx, 2 * dx, dim)
    ps, os_ = pe.Particles(dim, 1000.0, mass, 2 * dx), O.Scene(dim, 1000.0, mass, 2 * dx)
    for s in (ps, os_):
        s.fill_box((0.1, 0.1, 0.1 if dim == 3 else 0.0), 7, 6, 5 if dim == 3 else 1, dx)
        s.jitter_fluid(9, 0.05 * dx)
        s.fill_box_boundary((0.0, 0.0, 0.0), (0.6, 0.5, 0.5 if dim == 3 else 0.0), dx, 1)
        for j in range(5):
            wall = ((0.05, 0.1 + dx * j, 0.1 if dim == 3 else 0.0), 1e-4, (1.0 if j % 2 else -1.0, 0.0, 0.0))
            s.push_boundary_oriented(*wall) if isinstance(s, pe.Particles) else s.push_boundary(*wall)
    ps.recomputed_akinci_psi()
    os_.recompute_psi()
    p = pe.DfsphParams(kernel=kernel, adaptive_dt=False, particle_diameter=dx, max_density_iters=5,
                       max_divergence_iters=5)
    q = O.dfsph_default_params()
    q.kernel, q.adaptive_dt, q.particle_diameter, q.max_density_iters, q.max_divergence_iters = kernel, 0, dx, 5, 5
    o = O.DfsphWorld(os_, q)
    o.run(1.0 / 240.0, 4)
    for lanes in (0, 1, 8, 32):
        w = pe.DfsphWorld(ps, p)
        w.set_lanes(lanes)
        w.compute_density()
        w.compute_alpha()
        w.run(1.0 / 240.0, 4)
        for a, b, what in ((w.positions(), o.x(), "x"), (w.velocities(), o.v(), "v"), (w.densities(), o.rho(), "rho"),
                           (w.boundary_forces(), o.boundary_force(), "boundary force"), (w.alphas(), o.alpha(), "alpha")):
            assert_bits_equal(a, b, f"{lanes} lanes {what}")
        assert w.last_iterations() == o.iterations()
        w.close()

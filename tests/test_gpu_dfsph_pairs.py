"""What the divergence-free solver keeps of its pairs between passes changes no
bit: with the buffer and without it, through slip planes, positions set between
steps and changed parameters, and with lists that reach beyond the buffer."""
import numpy as np
import pytest

import physics_engine_rs as pe
from helpers import assert_bits_equal

pytestmark = pytest.mark.gpu

DX = 0.05


def _world(dim, lanes, spread=1.0, at=0.1, wall=0.7, neighbours=4, **kw):
    mass = pe.mass_calibrated_to_rest(1000.0, DX, 2 * DX, dim)
    p = pe.Particles(dim, 1000.0, mass, 2 * DX)
    p.fill_box((at, at, at if dim == 3 else 0.0), 10, 8, 9 if dim == 3 else 1, DX * spread)
    p.jitter_fluid(9, 0.05 * DX)
    p.fill_box_boundary((0.0, 0.0, 0.0), (wall + 0.05, wall, wall + 0.1 if dim == 3 else 0.0), DX, 1)
    for j in range(5):
        p.push_boundary_oriented((at - 0.05, at + DX * j, at if dim == 3 else 0.0), 1e-4, (1.0 if j % 2 else -1.0, 0.0, 0.0))
    p.recomputed_akinci_psi()
    w = pe.DfsphWorld(p, pe.DfsphParams(adaptive_dt=False, particle_diameter=DX, max_density_iters=5,
                                        max_divergence_iters=5, xsph_epsilon=0.05, **kw),
                      pe.WcsphConfig(max_neighbours=neighbours))  # few: the first build sizes the pool
    w.set_lanes(lanes)
    return w


def _same(a, b, what):
    for x, y, name in ((a.positions(), b.positions(), "x"), (a.velocities(), b.velocities(), "v"),
                       (a.densities(), b.densities(), "rho"), (a.alphas(), b.alphas(), "alpha"),
                       (a.boundary_forces(), b.boundary_forces(), "boundary force")):
        assert_bits_equal(x, y, f"{what} {name}")
    assert a.last_iterations() == b.last_iterations()


@pytest.mark.parametrize("dim,lanes", [(3, 0), (3, 1), (3, 8), (2, 32)])
def test_kept_pairs_change_nothing(dim, lanes):
    slip = {"free_slip_xmin": 0.11, "free_slip_ymax": 0.45}
    worlds = [_world(dim, lanes, **slip) for _ in range(2)]
    worlds[1].set_pair_weights(False)
    dt = 1.0 / 240.0
    for w in worlds:
        w.run(dt, 2)
    _same(*worlds, "steps")
    x = worlds[0].positions()
    x[:60] += np.array([0.004, -0.003, 0.0])
    for w in worlds:
        w.set_positions(x)  # lists and alpha stay those of the old positions
        w.run(dt, 1)
    _same(*worlds, "set positions")
    for w in worlds:
        w.set_positions(x)
        w.compute_alpha()
        w.run(dt, 2)
    _same(*worlds, "alpha again")
    worlds[0].set_pair_weights(False)
    worlds[1].set_pair_weights(True)
    for w in worlds:
        w.run(dt, 2)
    _same(*worlds, "switched")
    for w in worlds:
        w.close()


@pytest.mark.parametrize("lanes,spread", [(0, 1.08), (1, 1.1), (8, 1.12), (0, 1.15), (1, 1.2)])
def test_lists_beyond_the_buffer(lanes, spread):
    """Worlds made wider than the one they are set to: the pool, sized for the
    first state, then holds lists of up to 1.5 times the need, the buffer those
    of up to 1.25 times."""
    wide, direct = _world(3, lanes, spread, 0.35, 1.2), _world(3, lanes, 1.0, 0.35, 1.2)
    direct.set_pair_weights(False)
    for w in (wide, direct):
        w.set_positions(direct.positions())
        w.rebuild_neighbours()
        w.compute_density()
        w.compute_alpha()
        if w is wide:  # the buffer, which the poll after that call extended, as first allocated
            w.set_pair_weights(False)
            w.set_pair_weights(True)
        w.run(1.0 / 240.0, 2)
    _same(wide, direct, f"{spread} wide")
    wide.close()
    direct.close()


def test_lists_survive_a_pool_that_grows():
    """Particles that rush together outgrow the pool between two steps: the poll
    after the first step moves it, and the next step begins with its lists."""
    worlds = [_world(3, 0, 1.7, 0.45, 1.9, neighbours) for neighbours in (4, 2048)]
    dt = 1.0 / 240.0
    x = worlds[0].positions()
    n = 10 * 8 * 9
    v = np.zeros_like(x)
    v[:n] = (x[:n].mean(0) - x[:n]) * (0.17 / dt)
    for w in worlds:
        w.set_velocities(v)
        w.run(dt, 1)
        w.set_velocities(0.0 * v)
        w.run(dt, 2)
    _same(*worlds, "grown")
    for w in worlds:
        w.close()

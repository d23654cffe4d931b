"""The list build's shared-memory stage after the host moves particles: it is
sized for the new positions before they are built on, and worlds of different
stage sizes do not disturb each other."""
import numpy as np
import pytest

import oracle as O
import physics_engine_rs as pe
from helpers import assert_bits_equal, dam_break_params_pe, product_dam_break

pytestmark = pytest.mark.gpu

BOX = (0.4, 0.3, 0.3)


@pytest.mark.parametrize("precision", [pe.PRECISION_F64, pe.PRECISION_F32])
@pytest.mark.parametrize("pack", [1.0, 0.8, 0.5])
def test_stage_follows_host_positions(pack, precision):
    """Packed to half the spacing, a cell's union is several times the one the world was created with."""
    ps = product_dam_break(16, 14, 12, box=BOX)
    w = pe.WcsphWorld(ps, dam_break_params_pe(False), pe.WcsphConfig(precision=precision))
    w.run(1e-6, 1)
    a = ps.arrays()
    fluid = a["kind"] == 0
    x = a["x"].copy()
    x[fluid] = 0.1 + pack * (x[fluid] - 0.1)
    w.set_positions(x)
    w.set_velocities(a["v"])
    w.run(1e-7, 3)
    assert w.status() & pe.STATUS_SLOW_UNION == 0
    info = w.capacity_info()
    assert info["max_union"] <= info["union_capacity"]
    if precision == pe.PRECISION_F64:
        fresh = pe.WcsphWorld.from_arrays(dam_break_params_pe(False), 3, ps.rest_density, ps.mass, ps.h, x, a["v"],
                                          a["kind"], a["psi"])
        fresh.run(1e-7, 3)
        assert_bits_equal(w.positions(), fresh.positions(), "x")
        assert_bits_equal(w.velocities(), fresh.velocities(), "v")
        assert_bits_equal(w.densities(), fresh.densities(), "rho")
        fresh.close()
    w.close()


def test_worlds_of_different_stages_side_by_side():
    dense = product_dam_break(20, 20, 20, dx=0.01, box=BOX)
    big = pe.WcsphWorld(dense, dam_break_params_pe(False))
    alone = pe.WcsphWorld(dense, dam_break_params_pe(False))
    alone.run(1e-5, 4)
    ref = alone.positions()
    small = pe.WcsphWorld(product_dam_break(3, 3, 3, box=(0.1, 0.1, 0.1)), dam_break_params_pe(False))
    assert small.capacity_info()["union_capacity"] < big.capacity_info()["union_capacity"]
    for _ in range(4):
        big.run(1e-5, 1)
        small.run(1e-5, 1)
    assert_bits_equal(big.positions(), ref, "x")
    for w in (big, alone, small):
        w.close()


def _world_and_oracle(build, dim=3):
    mass = pe.mass_from_spacing(1000.0, 0.01, dim)
    ps, os_ = pe.Particles(dim, 1000.0, mass, 0.02), O.Scene(dim, 1000.0, mass, 0.02)
    build(ps)
    build(os_)
    return pe.WcsphWorld(ps, dam_break_params_pe(False)), O.World(os_, O.dam_break_params(materialize=False))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("count", [1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 97, 129])
def test_cell_populations_at_the_tile_edges(count, dim):
    """`count` particles in one cell (a chunk of 16, 32 and their neighbours; unions around multiples of 32
    candidates), a third of them boundary samples, with a second cell in reach."""
    rng = np.random.default_rng(count)
    x = rng.uniform(0.041, 0.079, (count + 7, 3))
    x[count:, 0] += 0.04
    if dim == 2:
        x[:, 2] = 0.0

    def build(s):
        for k, p in enumerate(x):
            s.push_boundary(tuple(p), 1e-6) if k % 3 == 2 else s.push_fluid(tuple(p), tuple(0.1 * p))

    w, o = _world_and_oracle(build, dim)
    w.run(1e-6, 2)
    o.run(1e-6, 2)
    for a, b, what in ((w.positions(), o.x(), "x"), (w.velocities(), o.v(), "v"), (w.densities(), o.rho(), "rho"),
                       (w.boundary_forces(), o.boundary_force(), "boundary force")):
        assert_bits_equal(a, b, what)
    for a, b in zip(w.neighbour_counts(), o.neighbour_counts()):
        np.testing.assert_array_equal(a.astype(np.int64), b)
    w.close()


def test_pairs_at_the_edge_of_the_support_are_kept():
    """Pairs a relative 1e-12 and 1e-3 inside the support, and as far outside, in random directions at random
    places of their cells: the half-precision filter of the list build loses none."""
    rng = np.random.default_rng(5)
    n = 1500
    place = np.stack(np.meshgrid(*[np.arange(12)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 0.2
    a = place + rng.uniform(0.0, 0.04, (n, 3))
    d = rng.normal(size=(n, 3))
    d[::5, 1:] = 0.0
    scale = rng.choice([1.0 - 1e-12, 1.0 - 1e-3, 1.0 + 1e-12, 1.0 + 1e-3], n)
    b = a + d / np.linalg.norm(d, axis=1, keepdims=True) * (0.04 * scale)[:, None]

    def build(s):
        for p, q in zip(a, b):
            s.push_fluid(tuple(p))
            s.push_fluid(tuple(q))

    w, o = _world_and_oracle(build)
    w.rebuild_grid()
    o.rebuild_grid()
    w.compute_density()
    counts = w.neighbour_counts()
    ref = o.neighbour_counts()
    np.testing.assert_array_equal(counts[0].astype(np.int64), ref[0])
    np.testing.assert_array_equal(counts[1].astype(np.int64), ref[1])
    inside = int(np.sum(ref[1] == np.max(ref[1])))
    assert n < inside < 2 * n  # both kinds are there
    w.close()

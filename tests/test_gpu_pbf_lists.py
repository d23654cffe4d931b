"""The constraint iterations' lists and passes of the Position Based Fluids step
reproduce the oracle bit for bit: unions of less than a warp's worth of
candidates, of one tile and of several, more than 32 particles a cell (several
chunks), predictions that leave their cells between two grids, oriented samples,
2-D, XSPH viscosity and tensile pressure, with 1 and with 8 lanes."""
import numpy as np
import pytest

import oracle as O
import physics_engine_rs as pe
from helpers import assert_bits_equal

pytestmark = pytest.mark.gpu

CASES = {  # dim, block, spacing, h, box, iterations, reuse, start speed
    "sparse": (3, (4, 3, 5), 0.05, 0.06, (0.6, 0.6, 0.6), 3, True, 0.0),
    "one tile": (3, (9, 8, 7), 0.05, 0.1, (0.8, 0.7, 0.9), 4, True, 1.0),
    "several tiles": (3, (9, 9, 10), 0.05, 0.17, (0.8, 0.8, 0.9), 4, True, 0.0),
    "several chunks": (3, (10, 9, 9), 0.05, 0.22, (0.9, 0.8, 0.9), 2, False, 0.0),
    "moving": (3, (8, 8, 8), 0.03, 0.1, (0.9, 0.9, 0.9), 9, True, 6.0),  # 0.6 of the spacing the masses are for
    "planar": (2, (14, 12, 1), 0.05, 0.21, (1.0, 0.9, 0.0), 5, True, 0.5),
}


@pytest.mark.parametrize("case", list(CASES))
def test_constraint_lists_bit_exact(case):
    dim, block, dx, h, box, iterations, reuse, speed = CASES[case]
    mass = pe.mass_from_spacing(1000.0, 0.05, dim)
    ps, os_ = pe.Particles(dim, 1000.0, mass, h), O.Scene(dim, 1000.0, mass, h)
    flat = 0.1 if dim == 3 else 0.0
    rng = np.random.default_rng(7)
    grid = np.stack(np.meshgrid(*(np.arange(k) for k in block), indexing="ij"), -1).reshape(-1, 3)
    x = np.array([0.1, 0.1, flat]) + dx * (grid + rng.uniform(-0.1, 0.1, grid.shape))
    v = rng.uniform(-speed, speed, x.shape)
    if dim == 2:
        x[:, 2] = v[:, 2] = 0.0
    for s in (ps, os_):
        for a, b in zip(x, v):
            s.push_fluid(tuple(a), tuple(b))
        s.fill_box_boundary((0.0, 0.0, 0.0), box, 0.05, 1)
        for j in range(4):
            wall = ((0.06, 0.1 + dx * j, flat), 1e-4, (1.0, 0.0, 0.0))
            s.push_boundary_oriented(*wall) if isinstance(s, pe.Particles) else s.push_boundary(*wall)
    g = (0.0, 0.0, -9.81) if dim == 3 else (0.0, -9.81, 0.0)
    p = pe.PbfParams(gravity=g, iterations=iterations, reuse_neighbours=reuse, art_pressure_k=1e-4, viscosity_eps=0.02)
    q = O.pbf_default_params()
    for k in pe.PbfParams._FIELDS:
        v = getattr(p, k)
        if k == "gravity":
            q.gravity[:] = v
        else:
            setattr(q, k, int(v) if isinstance(v, bool) else v)
    o = O.PbfWorld(os_, q)
    o.run(1.0 / 120.0, 3)
    for lanes in (0, 1, 8):
        w = pe.PbfWorld(ps, p)
        w.set_lanes(lanes)
        w.run(1.0 / 120.0, 3)
        for a, b, what in ((w.positions(), o.x(), "x"), (w.velocities(), o.v(), "v"), (w.densities(), o.rho(), "rho"),
                           (w.lambdas(), o.lam(), "lambda")):
            assert_bits_equal(a, b, f"{case}, {lanes} lanes, {what}")
        assert w.status() & ~pe.STATUS_SLOW_UNION == 0
        w.close()


def test_other_lane_counts_are_refused():
    ps = pe.Particles(3, 1000.0, pe.mass_from_spacing(1000.0, 0.05, 3), 0.1)
    ps.fill_box((0.1, 0.1, 0.1), 3, 3, 3, 0.05)
    w = pe.PbfWorld(ps, pe.PbfParams())
    for lanes in (2, 4, 32):
        with pytest.raises(pe.PeError):
            w.set_lanes(lanes)
    w.close()

"""The list build's shared-memory stage after the host moves particles: it is
sized for the new positions before they are built on, and worlds of different
stage sizes do not disturb each other."""
import numpy as np
import pytest

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

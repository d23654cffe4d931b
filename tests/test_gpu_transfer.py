"""State import and export: large copies by several threads through pinned
slots, small ones and pinned memory by one copy; every byte arrives, at sizes
that leave ragged parts and slots, from addresses of any alignment, and with
worlds used by several threads at once."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

import physics_engine_rs as pe
from helpers import dam_break_params_pe

pytestmark = pytest.mark.gpu

DX = 0.01


def _world(nx, ny):
    p = pe.Particles(2, 1000.0, pe.mass_from_spacing(1000.0, DX, 2), 2 * DX)
    p.fill_box((0.0, 0.0, 0.0), nx, ny, 1, DX)
    return pe.WcsphWorld(p, dam_break_params_pe(False))


def _round_trips(w, seed, pinned=False):
    rng = np.random.default_rng(seed)
    n = w.n
    for _ in range(2):
        if pinned:
            v = torch.empty(n, 3, dtype=torch.float64).pin_memory().numpy()
        else:
            v = np.empty(3 * n + 1)[1:].reshape(n, 3)  # 8 bytes past the allocator's alignment
        v[:] = rng.normal(size=(n, 3))
        x = w.positions() + rng.uniform(-1e-4, 1e-4, (n, 3)) * np.array([1.0, 1.0, 0.0])
        w.set_velocities(v)
        w.set_positions(x)
        assert np.array_equal(w.velocities(), v)
        assert np.array_equal(w.positions(), x)


# 48 kB; the last size of one copy (16 MB) and the first of several threads; 24 MB
# whose last slots and parts are ragged, and whose scalars (8 MB) are shared out too
@pytest.mark.parametrize("shape", [(50, 40), (699, 1000), (700, 1000), (1051, 1001)])
def test_round_trip(shape):
    w = _world(*shape)
    _round_trips(w, 1)
    _round_trips(w, 2, pinned=True)
    w.close()


def test_non_finite_input_is_refused_and_leaves_the_state():
    w = _world(801, 899)
    v = np.zeros((w.n, 3))
    w.set_velocities(v)
    v[-1, 2] = np.nan
    with pytest.raises(pe.PeError):
        w.set_velocities(v)
    assert not w.velocities().any()
    w.close()


def test_worlds_of_several_threads():
    worlds = [_world(801, 899 + k) for k in range(3)]
    with ThreadPoolExecutor(3) as pool:
        list(pool.map(_round_trips, worlds, range(3)))
    for w in worlds:
        w.close()

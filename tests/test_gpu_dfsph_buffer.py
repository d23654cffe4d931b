"""The buffer in which the divergence-free solver keeps its pairs: made by the first pass that fills it, not by
the creation of a world, and reached beyond where the tests of that path mean it to be."""
import pytest

import physics_engine_rs as pe
from test_gpu_dfsph_pairs import _same, _world

pytestmark = pytest.mark.gpu


def test_the_buffer_is_made_when_it_is_first_filled():
    by_step, by_alpha, off = (_world(3, 0) for _ in range(3))
    for w in (by_step, by_alpha, off):
        assert w.pair_weight_info() == {"in_use": False, "entries": 0, "short": False}
    off.set_pair_weights(False)
    by_alpha.compute_alpha()
    assert by_alpha.pair_weight_info()["in_use"]
    for w in (by_step, by_alpha, off):
        w.run(1.0 / 240.0, 2)
    info = by_step.pair_weight_info()
    assert info["in_use"] and info["entries"] > 0
    assert not off.pair_weight_info()["in_use"]
    _same(by_step, by_alpha, "made by a step and by alpha")
    _same(by_step, off, "with and without")
    for w in (by_step, by_alpha, off):
        w.close()


def test_an_empty_world_has_none():
    w = pe.DfsphWorld(pe.Particles(3, 1000.0, 1e-3, 0.1), pe.DfsphParams(adaptive_dt=False))
    w.run(1e-3, 1)
    assert not w.pair_weight_info()["in_use"]
    w.close()


def test_lists_do_reach_beyond_the_buffer():
    """The worlds of test_gpu_dfsph_pairs.test_lists_beyond_the_buffer, and more of their kind: made wider than
    the state they are set to, their pools hold that state's lists, their buffers (of 5/8 of the pool) not all of
    them. Some of each world's lists are kept then and some computed, with one lane a list and with several."""
    short = {0: 0, 1: 0, 8: 0, 32: 0}
    for lanes in short:
        direct = _world(3, lanes, 1.0, 0.35, 1.2)
        direct.set_pair_weights(False)
        x = direct.positions()
        worlds = [direct]
        for spread in (1.08, 1.1, 1.12, 1.15, 1.2):
            w = _world(3, lanes, spread, 0.35, 1.2)
            worlds.append(w)
            w.set_positions(x)
            w.rebuild_neighbours()
            w.compute_density()
            w.set_pair_weights(False)
            w.set_pair_weights(True)
            w.compute_alpha()
            info = w.pair_weight_info()
            assert info["in_use"] and info["entries"] > 0
            short[lanes] += info["short"]
        direct.rebuild_neighbours()
        direct.compute_density()
        direct.compute_alpha()
        for w in worlds:
            w.run(1.0 / 240.0, 2)
        for w in worlds[1:]:
            _same(w, direct, f"{lanes} lanes")
        for w in worlds:
            w.close()
    assert all(short.values()), short

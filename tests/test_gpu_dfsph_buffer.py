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

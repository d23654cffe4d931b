"""Inference's fused edge and node MLPs against the GEMMs that training uses, bit
for bit: both round at the same points and add in the same order, and with at
most one edge a node the message sums have no order to differ in. Node and edge
counts around a warp, a tile of 128 and a round of all tiles; nodes that are not
fluid (their features stay)."""
import numpy as np
import pytest

from physics_engine_rs.surrogate import Surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E", [(1, 0), (31, 31), (127, 5), (128, 128), (129, 129), (700, 511), (3000, 0), (57000, 33000),
                                 (90001, 90001)])
def test_fused_matches_gemms_bit_for_bit(n, E):
    rng = np.random.default_rng(n + E)
    s = Surrogate(seed=5)
    dst = np.sort(rng.choice(n, E, replace=False))
    row = np.searchsorted(dst, np.arange(n + 1)).astype(np.int32)
    src = rng.integers(0, n, E).astype(np.int32)
    f = rng.normal(size=(n, 8))
    s.set_graph(f, rng.normal(size=(E, 16)), row, src, (rng.uniform(size=n) < 0.7).astype(np.uint8))
    s.set_fused_edges(False)
    want = s.forward()
    s.set_fused_edges(True)
    for _ in range(2):
        got = s.forward()
        assert np.isfinite(got).all() and got.any()
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))

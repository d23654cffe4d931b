"""Training gradients are sums in a fixed order: the same bits from run to run."""
import numpy as np
import pytest

import surrogate_ref as S
from physics_engine_rs.surrogate import Surrogate
from test_oracle_surrogate import random_graph, random_params

pytestmark = pytest.mark.gpu


def _graph(n, E, hub=0.0, seed=11):
    """A random graph; a share `hub` of the edges comes from node 0."""
    rng = np.random.default_rng(seed)
    f, xe, dst, src, fluid, t = random_graph(rng, n, E)
    src = np.where(rng.random(E) < hub, 0, src).astype(np.int32)
    return f, xe, dst, src, fluid, t


def _net(n, graph, p, seed=1):
    s = Surrogate(seed=seed)
    s.set_params(p)
    _set(s, n, graph)
    return s


def _set(s, n, graph):
    f, xe, dst, src, fluid, t = graph
    s.set_graph(f, xe, np.searchsorted(dst, np.arange(n + 1)).astype(np.int32), src, fluid)
    s.set_targets(t)


def _params(seed=7):
    return {k: v.astype(np.float32) for k, v in random_params(np.random.default_rng(seed)).items()}


def _grads(s):
    s.train_step(0.0)
    return {k: v.copy() for k, v in s.get_params(grads=True).items()}


def _same(a, b):
    bad = [k for k in a if not np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32))]
    assert not bad, bad


SIZES = [(1000, 22000, 0.0), (1800, 60001, 0.0), (5003, 120000, 0.3), (15000, 330017, 0.0)]


@pytest.mark.parametrize("n,E,hub", SIZES)
def test_gradients_repeat(n, E, hub):
    g, p = _graph(n, E, hub), _params()
    s = _net(n, g, p)
    first = _grads(s)
    for _ in range(3):
        _same(first, _grads(s))
    _same(first, _grads(_net(n, g, p)))


def test_edges_are_ordered_again_for_a_new_graph():
    """A graph that replaces another, with as many edges, with fewer, and with none."""
    p = _params()
    s = _net(600, _graph(600, 5000), p)
    s.train_step(0.0)
    for n, E, hub, seed in ((600, 5000, 0.5, 12), (300, 1, 0.0, 13), (300, 0, 0.0, 14), (601, 4999, 0.0, 15)):
        g = _graph(n, E, hub, seed)
        _set(s, n, g)
        _same(_grads(s), _grads(_net(n, g, p)))


def _dyadic(rng, n, E, hub):
    """Weights, features and targets that are small multiples of 1/4, three weights an output: the sums of the
    forward pass are exact in any order, so no ReLU and no rounding depends on it."""
    p = {}
    for k, v in random_params(rng).items():
        if k.endswith(".b"):
            p[k] = rng.integers(-2, 3, v.shape) * 0.25
            continue
        p[k] = np.zeros(v.shape)
        for j in range(v.shape[1]):
            p[k][rng.integers(0, v.shape[0], 3), j] = rng.choice([-0.5, 0.5, 1.0], 3)
    dst = np.sort(rng.integers(0, n, E))
    src = np.where(rng.random(E) < hub, 0, rng.integers(0, n, E))
    f, xe = rng.integers(-4, 5, (n, 8)) * 0.25, rng.integers(-4, 5, (E, 16)) * 0.25
    graph = (f, xe, dst, src.astype(np.int32), rng.random(n) < 0.7, rng.integers(-8, 9, (n, 4)) * 0.25)
    return {k: v.astype(np.float32) for k, v in p.items()}, graph


@pytest.mark.parametrize("n,E,hub,seed", [(60, 600, 0.7, 1), (300, 2400, 0.0, 2), (1000, 9000, 0.3, 3), (33, 1, 0.0, 4)])
def test_source_side_gradients_match_the_oracle(n, E, hub, seed):
    """Sources with most of the edges, and with none. Bound: the last product's fp32 sum over n rows is off by at
    most n 2^-23 of it, and a bf16 rounding that a backward sum's last bit turns costs 2^-9 of one of 128 n
    elements (some of them: 1e-4); an edge left out or taken twice costs about 1 / sqrt(E), 1e-2."""
    p, graph = _dyadic(np.random.default_rng(seed), n, E, hub)
    f, xe, dst, src, fluid, t = graph
    s = _net(n, graph, p)
    s.train_step(0.0)
    g = s.get_params(grads=True)
    net = S.Net({k: v.astype(np.float64) for k, v in p.items()})
    _, _, ref = net.loss_and_grads(S.bf16(f), S.bf16(xe), dst, src, fluid, t)
    for k in ("hop1.edge.a.W", "hop1.edge.b.W", "hop2.edge.b.W", "enc.0.W", "enc.2.W"):
        off = np.linalg.norm(g[k].astype(np.float64) - ref[k]) / np.linalg.norm(ref[k])
        assert off <= n * 2.0**-23 + 1e-4, (k, off)

"""A network allocates what its path touches: nodes only for fused inference, a hop's layers for the GEMMs', all of
it for training; and any order of the three, on graphs that grow and shrink, gives a fresh network's bits."""
import numpy as np
import pytest

from physics_engine_rs.surrogate import Surrogate
from test_gpu_gradient_order import _graph, _params, _set

pytestmark = pytest.mark.gpu


def _fresh(p, n, graph, fused=True):
    s = Surrogate(seed=1)
    s.set_params(p)
    s.set_fused_edges(fused)
    _set(s, n, graph)
    return s


def _same(a, b, what):
    assert np.array_equal(np.asarray(a, np.float32).view(np.uint32), np.asarray(b, np.float32).view(np.uint32)), what


def test_inference_allocates_no_edge_buffers():
    import torch

    p, n, E = _params(), 20000, 400000
    s = _fresh(p, n, _graph(n, E))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s.forward()
    taken = before - torch.cuda.mem_get_info()[0]
    # 22 bytes a node and column with a quarter of headroom: 70 MB; the edges' activations alone are 512 MB
    assert taken < 200e6, taken


@pytest.mark.parametrize("order", ["fusf", "ufsu", "sfuf", "fsus"])
def test_any_order_of_inference_and_training(order):
    """f: fused inference, u: the layers' GEMMs, s: a training step's gradients; each on a graph of its own."""
    p = _params()
    # one edge a node at most: a fused message sum has one order
    sizes = [(900, 700), (300, 250), (2000, 1999), (1500, 0)]
    net = Surrogate(seed=1)
    net.set_params(p)
    for what, (n, E) in zip(order, sizes):
        f, xe, _, src, fluid, t = _graph(n, max(E, 1), seed=n)
        graph = (f, xe[:E], np.sort(np.random.default_rng(n).permutation(n)[:E]), src[:E], fluid, t)
        _set(net, n, graph)
        net.set_fused_edges(what != "u")
        ref = _fresh(p, n, graph, what != "u")
        if what == "s":
            net.train_step(0.0)
            ref.train_step(0.0)
            a, b = net.get_params(grads=True), ref.get_params(grads=True)
            for k in a:
                _same(a[k], b[k], (order, what, k))
        else:
            _same(net.forward(), ref.forward(), (order, what))
        # the same graph again, after the other paths have had their turn on it
        net.train_step(0.0)
        net.set_fused_edges(True)
        _same(net.forward(), _fresh(p, n, graph).forward(), (order, what, "again"))

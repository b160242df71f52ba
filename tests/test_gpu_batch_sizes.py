"""Batched mode at the edges of its working arrays: graphs of one node up to
the 16,384 limit, leaf sizes from the shallowest to the deepest quadtree, and
launch shapes whose CTAs hold all, some or few of a graph's arrays in shared
memory. The kick is compared with an FP64 direct sum (the tolerance of
test_gpu_batch.py: FP32 positions scaled to the box and order-8 expansions),
the states after ticks with the first shape's, bit for bit."""

import importlib

import numpy as np
import pytest

import helpers as H

B = importlib.import_module("d3-force-wasm_b200.batch")
pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 31, 65, 257, 1025, 4097, 9001, 16383, 16384)


def _graphs():
    rng = np.random.default_rng(11)
    graphs, starts = [], []
    for n in SIZES:
        m = 2 * n if n > 1 else 0
        src = rng.integers(0, max(n, 1), m)
        tgt = (src + 1 + rng.integers(0, max(n - 1, 1), m)) % n
        graphs.append((n, src.astype(np.uint32), tgt.astype(np.uint32)))
        side = 10 * np.sqrt(n)
        # one half uniform, one half in a dense corner: uneven leaves
        x, y = rng.random(n) * side, rng.random(n) * side
        x[::2] *= 0.3
        y[::2] *= 0.3
        starts.append((x, y))
    return graphs, starts


@pytest.mark.parametrize("leaf", [2, 16, 256])
def test_gpu_batch_sizes_and_shapes(gcore, leaf):
    graphs, starts = _graphs()
    states = []
    for threads, per_sm in ((1024, 1), (256, 1), (512, 2)):
        b = B.Batch(gcore, graphs, starts)
        try:
            b.set_shape(threads, per_sm, leaf)
            kick, alpha = b.kick()
            rms = B.graph_rms(b, kick, alpha, range(1, len(SIZES)))
            assert rms.max() < 1e-4, (threads, per_sm, rms)
            assert np.all(kick[0] == 0)  # a lone node feels nothing
            b.run(3, graph=False)
            states.append(np.concatenate([a.view(np.uint32) for a in b.read()]))
        finally:
            b.close()
    assert np.array_equal(states[0], states[1]) and np.array_equal(states[0], states[2])


def test_gpu_batch_coincident_and_far_nodes(gcore):
    """Coincident nodes take the hashed jiggle and come apart; a far outlier
    leaves nearly every node in one cell of both grids; all stay finite."""
    n = 700
    rng = np.random.default_rng(3)
    x, y = rng.random(n) * 50, rng.random(n) * 50
    x[1], y[1] = x[0], y[0]
    x[2] = x[0]  # one zero delta
    x[-1], y[-1] = 4e6, -3e6
    z = np.zeros(0, np.uint32)
    b = B.Batch(gcore, [(n, z, z)], [(x, y)])
    try:
        b.run(2, graph=True)
        state = b.read()
    finally:
        b.close()
    assert all(np.all(np.isfinite(a)) for a in state)
    assert state[0][0] != state[0][1] or state[1][0] != state[1][1]

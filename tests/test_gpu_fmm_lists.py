"""The fast many-body passes where their shapes turn: orders at which the
lanes per source and the sources side by side change, lists past the shared
ones (a dense cluster beside sparse leaves) and past the first pools, long P2P
lists in segments, leaves of
16, 17 and 32 points and of more than a warp's chunk, one leaf as the whole
tree. Positions equal the oracle's bit for bit."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


def _layout(kind, n):
    rng = np.random.default_rng(n)
    x, y = rng.random(n) * 3000, rng.random(n) * 3000
    if kind == "cluster":  # nine in ten within a hundredth of the square
        k = 9 * n // 10
        x[:k], y[:k] = 1700 + 30 * rng.random(k), 1450 + 30 * rng.random(k)
    if kind == "far":  # one node far from the rest: a leaf child of the root
        x[0], y[0] = 4e5, 4e5
    if kind == "beside":  # nineteen in twenty in a cluster among sparse leaves
        k = 19 * n // 20
        x[:k], y[:k] = 1500 + 120 * rng.standard_normal(k), 1500 + 120 * rng.standard_normal(k)
        x[:40] = x[0] + 0.3 * rng.random(40)
        y[:40] = y[0] + 0.3 * rng.random(40)
    if kind == "clump":  # 77 nodes on one spot: three chunks of a source leaf
        x[:77], y[:77] = 1234.5, 777.25
    if kind == "blocks":  # leaves of exactly 16, 17 and 32 points on an 8 x 8 grid
        counts = [(16, 17, 32)[i % 3] for i in range(64)]
        at = np.repeat(np.arange(64), counts)[:n]
        x = (at % 8 + 0.1 + 0.8 * rng.random(len(at))) * 400
        y = (at // 8 + 0.1 + 0.8 * rng.random(len(at))) * 400
    return x, y


def _run(ocore, gcore, kind, n, ticks, order=None, opening=None, dmax=None):
    x, y = _layout(kind, n)
    kw = {k: v for k, v in (("order", order), ("opening", opening)) if v is not None}

    def setup(core):
        nodes = pkg.Nodes(len(x), x=list(x), y=list(y))
        sim = pkg.forceSimulation(nodes, core=core)
        mb = pkg.forceManyBody()
        if dmax is not None:
            mb.distanceMax(dmax)
        sim.force("charge", mb)
        sim.precision("fast", **kw)
        return nodes, sim
    P.run_pair(setup, ocore, gcore, ticks)


@pytest.mark.parametrize("order", [1, 2, 3, 5, 7, 9, 10, 11, 15, 16, 20, 23, 24])
def test_gpu_fmm_orders(ocore, gcore, order):
    _run(ocore, gcore, "uniform", 2000, 2, order=order)


@pytest.mark.parametrize("kind,n,dmax", [("cluster", 20001, None), ("cluster", 20001, 90.0),
                                         ("far", 3000, None), ("clump", 3000, None),
                                         ("blocks", 1386, None), ("uniform", 32, None),
                                         ("uniform", 33, None), ("uniform", 17, None)])
def test_gpu_fmm_shapes(ocore, gcore, kind, n, dmax):
    _run(ocore, gcore, kind, n, 3, dmax=dmax)


@pytest.mark.parametrize("kind,n,dmax", [("beside", 9000, None), ("beside", 40001, 700.0),
                                         ("beside", 40001, None)])
def test_gpu_fmm_long_lists(ocore, gcore, kind, n, dmax):
    """Leaves beside a dense cluster (lists of hundreds of leaves; clumps closer
    than distanceMin in it, whose groups go pair by pair), with leaves of up to
    16 and of more targets: the second tick on has the room for their terms."""
    _run(ocore, gcore, kind, n, 4, dmax=dmax)


def test_gpu_fmm_pools_grow(ocore, gcore):
    """A wide opening: more list entries a cell than the first pools hold."""
    _run(ocore, gcore, "uniform", 9000, 2, opening=4.0)

"""The exact link pass on both of its paths, bit for bit against the oracle:
the one-block pass (up to 7,000 nodes) and the message pass, at their
boundary, with long dependency chains (a hub), repeated links, several
iterations, and passes that end serially (a link from a node to itself, linked
nodes at one position)."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


def _links(kind, n, rng):
    if kind == "hub":  # every link on node 0: one link per level
        k = min(n - 1, 600)
        return np.zeros(k, np.int64), 1 + np.arange(k)
    if kind == "path":
        return np.arange(n - 1), np.arange(1, n)
    m = 3 * n
    src = rng.integers(0, n, m)
    tgt = (src + 1 + rng.integers(0, n - 1, m)) % n
    if kind == "repeated":  # a few pairs over and over, in both directions
        k = rng.integers(0, 5, m)
        src, tgt = np.where(k % 2, k % n, (k + 1) % n), np.where(k % 2, (k + 1) % n, k % n)
        src, tgt = src[:200], tgt[:200]
    if kind == "self":
        tgt[m // 2] = src[m // 2]
    return src, tgt


def _setup(n, kind, iterations, coincident=False):
    rng = np.random.default_rng([n, iterations, len(kind)])
    x, y = rng.random(n) * 500, rng.random(n) * 500
    src, tgt = _links(kind, n, rng)
    if coincident:
        x[tgt[3]], y[tgt[3]] = x[src[3]], y[src[3]]
    # nodes past the last linked one keep their velocity
    v = rng.standard_normal((2, n))

    def setup(core):
        nodes = pkg.Nodes(n, x=x, y=y, vx=v[0], vy=v[1])
        sim = pkg.forceSimulation(nodes, core=core)
        sim.force("link", pkg.forceLink(src, tgt).iterations(iterations))
        return nodes, sim

    return setup


@pytest.mark.parametrize("n", [2, 33, 1000, 7000, 7001, 20011])
@pytest.mark.parametrize("iterations", [1, 3])
def test_gpu_link_random(ocore, gcore, n, iterations):
    P.run_pair(_setup(n, "random", iterations), ocore, gcore, 3)


@pytest.mark.parametrize("n", [700, 7500])
@pytest.mark.parametrize("kind", ["hub", "path", "repeated", "self"])
def test_gpu_link_chains(ocore, gcore, n, kind):
    P.run_pair(_setup(n, kind, 2), ocore, gcore, 2)


@pytest.mark.parametrize("n", [500, 9000])
def test_gpu_link_jiggle_pass_is_serial(ocore, gcore, n):
    # the coincident pair makes tick 1 a serial pass; the next ones are not
    P.run_pair(_setup(n, "random", 1, coincident=True), ocore, gcore, 3)

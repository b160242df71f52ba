"""The exact many-body force on its size-dependent paths, bit for bit against
the oracle: the one-block tree build (up to 1,024 points), the one-block
accumulation (384), the warp-per-target traversal (7,000) and the paths past
them; runs of points equal in the sort word's bits, nodes with a NaN
coordinate, opening angles whose visits overflow the warp's stack, a finite
distanceMax, zero and NaN strengths."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    x, y = rng.random(n) * 1000 - 300, rng.random(n) * 1000 - 700
    if kind == "pairs":  # neighbours 1e-12 apart: equal in the key's top bits
        h = min(n // 16, 60)  # (each hangs a chain of 40 cells; the buffers hold 4 n)
        x[h:2 * h] = x[:h] + 1e-12 * (rng.random(h) - 0.5)
        y[h:2 * h] = y[:h] + 1e-12 * (rng.random(h) - 0.5)
        x[:3], y[:3] = x[0], y[0]  # and three on one spot
    if kind == "grid":  # zero deltas everywhere
        x, y = 12.0 * (np.arange(n) % 31), 12.0 * (np.arange(n) // 31)
    if kind == "corner":  # the box's far corner is a point of the largest key
        x[-1], y[-1] = x.max() + 1, y.max() + 1
    return x, y


def _setup(n, kind, theta=0.9, dmax=None, strength=None, nan=False):
    rng = np.random.default_rng([n, len(kind)])
    x, y = _points(kind, n, rng)

    def setup(core):
        nodes = pkg.Nodes(n, x=x, y=y, vx=np.zeros(n), vy=np.zeros(n))
        sim = pkg.forceSimulation(nodes, core=core)
        charge = pkg.forceManyBody().theta(theta)
        if dmax:
            charge.distanceMax(dmax)
        if strength:
            charge.strength(strength)
        sim.force("charge", charge)
        if nan:
            nodes.x[1::7] = np.nan
        return nodes, sim

    return setup


@pytest.mark.parametrize("n", [1, 2, 31, 64, 65, 384, 385, 1000, 1024, 1025, 3000, 7000, 7001])
@pytest.mark.parametrize("kind", ["uniform", "pairs", "corner"])
def test_gpu_many_body_sizes(ocore, gcore, n, kind):
    P.run_pair(_setup(n, kind), ocore, gcore, 2)


@pytest.mark.parametrize("n", [300, 1024, 2500])
def test_gpu_many_body_zero_deltas(ocore, gcore, n):
    P.run_pair(_setup(n, "grid"), ocore, gcore, 2)


@pytest.mark.parametrize("n", [60, 900, 2500])
def test_gpu_many_body_nan_nodes(ocore, gcore, n):
    P.run_pair(_setup(n, "uniform", nan=True), ocore, gcore, 1)


@pytest.mark.parametrize("theta", [0.02, 0.3, 2.0])
def test_gpu_many_body_opening_angles(ocore, gcore, theta):
    # at 0.02 nearly every cell is opened
    P.run_pair(_setup(4000, "uniform", theta=theta), ocore, gcore, 1)


def test_gpu_many_body_options(ocore, gcore):
    P.run_pair(_setup(1500, "uniform", dmax=250.0), ocore, gcore, 2)
    P.run_pair(_setup(700, "uniform", strength=lambda i: 0.0 if i % 3 else -30.0 - i), ocore, gcore, 2)
    P.run_pair(_setup(700, "uniform", strength=lambda i: float("nan") if i == 5 else -30.0), ocore,
               gcore, 1)


def test_gpu_many_body_after_shrinking(ocore, gcore):
    """A simulation that was larger before keeps its larger buffers."""
    def setup(core):
        nodes, sim = _setup(9000, "uniform")(core)
        sim.tick()
        rng = np.random.default_rng(5)
        small = pkg.Nodes(800, x=rng.random(800) * 100, y=rng.random(800) * 100)
        sim.nodes(small)
        return small, sim

    P.run_pair(setup, ocore, gcore, 2)

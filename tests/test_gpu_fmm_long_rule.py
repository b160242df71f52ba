"""Which plain runs take their long P2P lists in segments: those whose longest
list of the run before pays for it, few cells and many (the fast many-body
pass alone: layouts whose longest lists are far from either line). Bit for bit
against the oracle, on the run that has the segments' room too."""

import numpy as np
import pytest

import helpers as H
import parity as P
import test_gpu_fmm_lists as T

pkg = H.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, n, segments", [
    ("uniform", 20000, False),   # few cells, short lists
    ("cluster", 20001, True),    # few cells, lists of hundreds of leaves
    ("uniform", 80000, False),   # more cells
    ("cluster", 60000, True)])
def test_gpu_fmm_long_lists_by_their_length(ocore, gcore, kind, n, segments):
    x, y = T._layout(kind, n)
    pairs = []
    for core in (ocore, gcore):
        nodes = pkg.Nodes(n, x=x, y=y)
        sim = pkg.forceSimulation(nodes, core=core)
        sim.force("charge", pkg.forceManyBody())
        sim.precision("fast")
        pairs.append((nodes, sim))
    try:
        for t in range(3):
            for nodes, sim in pairs:  # (a tick blows the cluster up: the start again)
                nodes.x[:], nodes.y[:], nodes.vx[:], nodes.vy[:] = x, y, 0, 0
                sim.tick(1)
            d = P.first_difference(pairs[0][0], pairs[1][0])
            assert d is None, "tick %d: %s" % (t, d)
            taken = gcore.sim_stat(pairs[1][1].ctx.h, 38)
            assert (taken > 0) == (segments and t > 0), (t, taken)
    finally:
        for _, sim in pairs:
            sim.close()


def test_gpu_fmm_short_long_lists_are_left_alone(gcore):
    """A clustered layout whose longest list (some 80 source leaves) does not
    pay for the two launches: no segments on any tick."""
    n = 6001
    rng = np.random.default_rng(n)
    side = 10 * np.sqrt(n)
    label = rng.integers(0, 16, n)
    sigma = side * (0.02 + 0.06 * rng.random(16))
    x = (rng.random(16) * side)[label] + sigma[label] * rng.standard_normal(n)
    y = (rng.random(16) * side)[label] + sigma[label] * rng.standard_normal(n)
    nodes = pkg.Nodes(n, x=x, y=y)
    sim = pkg.forceSimulation(nodes, core=gcore)
    sim.force("charge", pkg.forceManyBody())
    sim.precision("fast")
    try:
        for _ in range(4):
            sim.tick(1)
            assert gcore.sim_stat(sim.ctx.h, 38) == 0
    finally:
        sim.close()

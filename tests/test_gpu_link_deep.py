"""Link chains of tens of thousands of levels go by messages to their end: the
wait of a link far down is not cut short while the links before it advance
(a pass that gave up would be run serially, with the same bits)."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, n, iterations", [("path", 20000, 1), ("path", 60000, 1), ("hub", 13001, 2)])
def test_gpu_link_deep_chain_is_not_cut_short(ocore, gcore, kind, n, iterations):
    rng = np.random.default_rng([n, iterations])
    x, y = rng.random(n) * 500, rng.random(n) * 500
    i = np.arange(n - 1)
    src, tgt = (i, i + 1) if kind == "path" else (0 * i, i + 1)
    pairs = []
    for core in (ocore, gcore):
        nodes = pkg.Nodes(n, x=x, y=y)
        sim = pkg.forceSimulation(nodes, core=core)
        sim.force("link", pkg.forceLink(src, tgt).iterations(iterations))
        pairs.append((nodes, sim))
    try:
        for t in range(2):
            for _, sim in pairs:
                sim.tick(1)
            d = P.first_difference(pairs[0][0], pairs[1][0])
            assert d is None, "tick %d: %s" % (t, d)
            # the pass met no jiggle and did not give up
            assert gcore.sim_stat(pairs[1][1].ctx.h, 5) == 0
            assert gcore.sim_stat(pairs[1][1].ctx.h, 4) == n - 1  # levels
    finally:
        for _, sim in pairs:
            sim.close()

"""New link sets between ticks: the messages of a plan's first pass start
empty although the memory held another plan's, bit for bit against the
oracle."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, plans", [(7001, 12), (20011, 36)])
def test_gpu_link_new_set_before_every_tick(ocore, gcore, n, plans):
    rng = np.random.default_rng([n, plans])
    x, y = rng.random(n) * 500, rng.random(n) * 500
    v = rng.standard_normal((2, n))
    pairs = []
    for core in (ocore, gcore):
        nodes = pkg.Nodes(n, x=x, y=y, vx=v[0], vy=v[1])
        pairs.append((nodes, pkg.forceSimulation(nodes, core=core)))
    m = 3 * n
    try:
        for k in range(plans):
            src = rng.integers(0, n, m)
            tgt = (src + 1 + rng.integers(0, n - 1, m)) % n
            for nodes, sim in pairs:
                sim.force("link", pkg.forceLink(src, tgt))
                sim.tick(1)
            d = P.first_difference(pairs[0][0], pairs[1][0])
            assert d is None, "plan %d: %s" % (k, d)
    finally:
        for _, sim in pairs:
            sim.close()

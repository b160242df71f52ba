"""Exact collide's guess by a warp (up to 8,192 nodes) and by a thread, and the
turns' chain: node counts around the line and below a warp, walks past the
warp's list (wide radii), heads past the guess's capacity (the serial loop),
mixed, zero and negative radii, NaN nodes. Positions equal the oracle's bit for
bit at every tick."""

import numpy as np
import pytest

import helpers as H
import parity as P

pkg = H.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,radius", [
    (2, 3, (2, 2)), (31, 60, (1, 8)), (1025, 200, (0, 6)), (3001, 300, (-2, 5)),
    (4000, 900, (1, 60)), (2000, 120, (6, 9)), (8192, 900, (4, 6)), (8193, 900, (4, 6))])
def test_gpu_collide_guess(ocore, gcore, n, side, radius):
    rng = np.random.default_rng(n)
    x, y = rng.random(n) * side, rng.random(n) * side
    r = radius[0] + rng.random(n) * (radius[1] - radius[0])

    def setup(core):
        nodes = pkg.Nodes(n, x=list(x), y=list(y))
        sim = pkg.forceSimulation(nodes, core=core)
        sim.force("collide", pkg.forceCollide().radius(lambda i: float(r[i])))
        if n > 100:
            nodes.x[n // 3] = float("nan")
        return nodes, sim
    P.run_pair(setup, ocore, gcore, 4)

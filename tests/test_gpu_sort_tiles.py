"""The device sort at its tiles' edges (2,048 keys), at the most one block takes
(8,192) and one more, with counts that come from
many tiles before (more than one read of the look-back), all keys of a pass
equal (the copy pass) and NaN nodes (the partition): fast many-body and fast
collide order their sums by it, so positions equal the oracle's bit for bit."""

import pytest

import helpers as H
import parity as P

pkg, sc = H.pkg, H.scenarios
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(1, 9.0), (2, 9.0), (2047, 400.0), (2048, 1e-3), (2049, 400.0),
                                      (8191, 900.0), (8192, 900.0), (8193, 900.0),
                                      (10240, 900.0), (10241, 900.0), (40961, 3000.0),
                                      (300001, 8000.0)])
def test_gpu_sort_tiles(ocore, gcore, n, spread):
    def setup(core):
        rnd = sc.generator(n)
        xs = [rnd() * spread for _ in range(n)]
        ys = [rnd() * spread for _ in range(n)]
        nodes = pkg.Nodes(n, x=xs, y=ys)
        sim = pkg.forceSimulation(nodes, core=core)
        sim.force("charge", pkg.forceManyBody())
        sim.force("collide", pkg.forceCollide(4))
        sim.precision("fast")
        if n > 2:
            nodes.x[n // 2] = float("nan")
            nodes.y[n - 1] = float("nan")
        return nodes, sim
    P.run_pair(setup, ocore, gcore, 1 if n > 100000 else 3)

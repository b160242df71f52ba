"""The plain FMM's list build when its waits run out (D3_LISTS_WAIT_NS=0: each
at once): a launch a level then gives the same lists. Bit for bit against the
oracle, in a process of its own (the limit is read once)."""

import os
import subprocess
import sys

import pytest

import helpers as H

pytestmark = pytest.mark.gpu

RUN = r"""
import sys
sys.path.insert(0, {tests!r})
import helpers as H, parity as P, test_gpu_fmm_lists as T
pkg = H.pkg
cores = H.oracle_core(), pkg.cuda_core()
for kind, n, dmax, opening in {cases!r}:
    x, y = T._layout(kind, n)
    pairs = []
    for core in cores:
        nodes = pkg.Nodes(len(x), x=list(x), y=list(y))
        sim = pkg.forceSimulation(nodes, core=core)
        mb = pkg.forceManyBody()
        if dmax is not None:
            mb.distanceMax(dmax)
        sim.force("charge", mb)
        sim.precision("fast", **({{}} if opening is None else {{"opening": opening}}))
        pairs.append((nodes, sim))
    for t in range(3):
        for _, sim in pairs:
            sim.tick(1)
        d = P.first_difference(pairs[0][0], pairs[1][0])
        assert d is None, (kind, n, t, d)
    again = cores[1].sim_stat(pairs[1][1].ctx.h, 29)
    assert {redone} == (again > 0), (kind, n, again)
"""
CASES = [("uniform", 2000, None, None), ("cluster", 20001, None, None), ("cluster", 20001, 90.0, None),
         ("beside", 40001, None, None), ("uniform", 9000, None, 4.0)]


@pytest.mark.parametrize("limit", ["0", None])
def test_gpu_fmm_lists_without_waits(limit):
    env = dict(os.environ)
    if limit is not None:
        env["D3_LISTS_WAIT_NS"] = limit
    code = RUN.format(tests=os.path.dirname(os.path.abspath(__file__)), cases=CASES, redone=limit == "0")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=env, cwd=H.ROOT)

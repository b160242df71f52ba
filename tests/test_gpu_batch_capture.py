"""Batched runs long enough to be captured in a CUDA graph (GRAPH_TICKS and
more) against the same ticks launched one by one, at several launch shapes and
split into runs in several ways: the same bits."""

import importlib
import re

import numpy as np
import pytest

import helpers as H
import test_stream_order as S

B = importlib.import_module("d3-force-wasm_b200.batch")
FEWEST = int(re.search(r"GRAPH_TICKS = (\d+);", S.source("batch.cu")).group(1))


def test_smoke_captures_its_run():
    with open(H.ROOT + "/__graft_entry__.py") as f:
        assert int(re.search(r"b\.run\((\d+), graph=True\)", f.read()).group(1)) >= FEWEST


@pytest.mark.gpu
def test_gpu_batch_captured_runs_equal_plain_ones(gcore):
    graphs = B.batch_workload(24, seed=5, nmax=4096)
    total = 2 * FEWEST + 5
    out = []
    for shape, runs in (((256, 1, 16), [(total, False)]),
                        ((256, 1, 16), [(total, True)]),
                        ((1024, 1, 16), [(FEWEST, True), (FEWEST + 5, True)]),
                        ((512, 2, 16), [(5, True), (FEWEST, True), (FEWEST, False)]),
                        ((1024, 1, 16), [(1, False)] * 3 + [(total - 3, True)])):
        b = B.Batch(gcore, graphs)
        try:
            b.set_shape(*shape)
            for ticks, graph in runs:
                b.run(ticks, graph=graph)
            out.append(np.concatenate([a.view(np.uint32) for a in b.read()]))
        finally:
            b.close()
    for k in range(1, len(out)):
        assert np.array_equal(out[0], out[k]), k

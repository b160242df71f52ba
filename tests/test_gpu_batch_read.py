"""Batched mode's read at the sizes where it turns to several threads (48 MB)
and at the edges of their pieces (512 KB): what all four arrays read at once give
equals the start positions, and after a tick the arrays read one by one (each
under the line: the plain copy), also from two threads at once."""

import ctypes
import importlib
import threading

import numpy as np
import pytest

B = importlib.import_module("d3-force-wasm_b200.batch")
pytestmark = pytest.mark.gpu

F32P = ctypes.POINTER(ctypes.c_float)


def _one(batch, k):
    out = np.full(batch.nodes, np.nan, np.float32)
    args = [None] * 4
    args[k] = out.ctypes.data_as(F32P)
    assert batch.lib.batch_read(batch.h, *args) == 0
    return out


@pytest.mark.parametrize("nodes", [3145727, 3145728, 3145729, 3276801, 4000001])
def test_gpu_batch_read_pieces(gcore, nodes):
    rng = np.random.default_rng(nodes)
    none = np.zeros(0, np.uint32)
    counts = [16384] * (nodes // 16384) + ([nodes % 16384] if nodes % 16384 else [])
    starts = [(rng.random(n) * 2000, rng.random(n) * 2000) for n in counts]
    batch = B.Batch(gcore, [(n, none, none) for n in counts], positions=starts)
    try:
        x, y, vx, vy = batch.read()
        assert np.array_equal(x, np.concatenate([s[0] for s in starts]).astype(np.float32))
        assert np.array_equal(y, np.concatenate([s[1] for s in starts]).astype(np.float32))
        assert not vx.any() and not vy.any()
        batch.run(1)
        got = [None, None]

        def read(i):
            got[i] = batch.read()
        threads = [threading.Thread(target=read, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(4):
            want = _one(batch, k)
            assert np.array_equal(got[0][k], want) and np.array_equal(got[1][k], want)
    finally:
        batch.close()

"""The tensor-core form's long lists: sparse nodes beside dense clusters, whose
P2P and W lists run to many segments and whose walks pass most of the tree,
leaves of more points than a segment's sums hold, and the tile counts around
one tile an SM; RMS against an FP64 direct sum, at test_gpu_fast_tc.py's
tolerance, and two runs with the same bits."""

import importlib

import numpy as np
import pytest

import helpers as H

pkg = H.pkg
acc = importlib.import_module("d3-force-wasm_b200.accuracy")
pytestmark = pytest.mark.gpu


def _layout(kind, n, rng):
    x, y = rng.random(n) * 1e4, rng.random(n) * 1e4
    # (no layout so dense that separated cells are nearer than distanceMin 1:
    # the form's far field has no clamp there)
    if kind == "cluster":  # nine in ten within one part in a hundred of the square
        k = 9 * n // 10
        x[:k] = 5003 + 60 * rng.standard_normal(k)
        y[:k] = 4997 + 60 * rng.standard_normal(k)
    if kind == "rings":  # clusters of falling width, one inside the other
        r = 5000 * 0.5 ** rng.integers(0, 6, n) * (0.6 + 0.4 * rng.random(n))
        t = rng.random(n) * 2 * np.pi
        x, y = 5000 + r * np.cos(t), 5000 + r * np.sin(t)
    if kind == "clump":  # 150 nodes on one spot: a leaf past every split
        x[:150], y[:150] = 1234.5, 777.25
    return x, y


@pytest.mark.parametrize("kind,n", [("cluster", 2001), ("cluster", 30000), ("rings", 9000),
                                    ("rings", 120000), ("clump", 4000), ("uniform", 150000),
                                    ("uniform", 260000)])
def test_gpu_tc_long_lists(gcore, kind, n):
    rng = np.random.default_rng(n)
    xs, ys = _layout(kind, n, rng)
    kick, alpha = acc.many_body_kick(pkg, gcore, xs, ys, form="bf16x3")
    again, _ = acc.many_body_kick(pkg, gcore, xs, ys, form="bf16x3")
    assert np.array_equal(kick, again)
    tg = acc.sample_targets(xs, ys, 1024)
    ref = acc.direct_kick(xs, ys, np.full(n, -30.0 * alpha), tg)
    assert acc.rms(kick, ref, tg) <= 1e-5

"""Which reads of a batch pin slots for themselves: those into memory that was
never touched, where one thread's page faults cost more than the pinning."""

import ctypes
import importlib
import mmap
import subprocess

import numpy as np
import pytest

import test_stream_order as S

HARNESS = r"""
#include <cstring>
#include "pages.cuh"
using d3::untouched_bytes;
static bool near(size_t a, size_t b, size_t by) { return a <= b + by && b <= a + by; }
int main() {
  const size_t n = 64u << 20;
  char *p = (char *)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) return 100;
  madvise(p, n, MADV_NOHUGEPAGE);
  if (untouched_bytes(p, n) != n) return 1;
  if (untouched_bytes(p + 3, n - 5) != n - 5) return 2;  // no need of aligned ends
  memset(p, 1, n / 2);
  if (!near(untouched_bytes(p, n), n / 2, n / 16)) return 3;
  memset(p, 1, n);
  if (untouched_bytes(p, n) != 0) return 4;
  if (untouched_bytes(p + 5, 100) || untouched_bytes(p, 0)) return 5;  // less than a page
  munmap(p, n);
  return untouched_bytes(p, n) ? 6 : 0;  // the kernel does not say: none
}
"""


def test_untouched_bytes(tmp_path):
    (tmp_path / "t.cc").write_text(HARNESS)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-x", "c++", "-I", S.CSRC, str(tmp_path / "t.cc"), "-o", exe])
    assert subprocess.run([exe]).returncode == 0


def test_slots_are_pinned_for_untouched_memory_only():
    read = S.source("batch.cu")
    read = read[read.index("bool read("):read.index("~Reader()")]
    assert "!workers_ && (untouched < READ_MIN || !reserve())" in read


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["touched first", "untouched first"])
def test_gpu_reads_into_touched_and_untouched_memory(gcore, order):
    B = importlib.import_module("d3-force-wasm_b200.batch")
    rng = np.random.default_rng(3)
    graphs = []
    for _ in range(196):  # 49 MB of state
        n = 16384
        src = rng.integers(0, n, n)
        graphs.append((n, src.astype(np.uint32), ((src + 1 + rng.integers(0, n - 1, n)) % n).astype(np.uint32)))
    b = B.Batch(gcore, graphs)
    try:
        b.run(1)
        out = []
        for kind in ("touched", "untouched", "touched")[order != "touched first":]:
            maps = [mmap.mmap(-1, 4 * b.nodes) for _ in range(4)]
            views = [np.frombuffer(m, np.float32) for m in maps]
            if kind == "touched":
                for v in views:
                    v[:] = np.nan
            C = importlib.import_module("d3-force-wasm_b200.core")
            C.check(b.lib.batch_read(b.h, *[v.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for v in views]))
            out.append(np.concatenate([v.view(np.uint32) for v in views]))
        assert all(np.array_equal(out[0], o) for o in out[1:])
        assert np.isfinite(out[0].view(np.float32)).all()
    finally:
        b.close()

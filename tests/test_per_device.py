"""A kernel's shared-memory attribute belongs to the device that was current
when it was set: it is set on every device a process uses, not once in the
process, and a launch that another path could stand in for is checked."""

import re
import subprocess

import pytest

import test_stream_order as S

HARNESS = r"""
#include <cstdio>
#include "per_device.cuh"
int main() {
  d3::PerDevice p;
  int calls[2] = {0, 0};
  auto works = [&](int d) { return p(d, [&, d] { ++calls[d]; return true; }); };
  auto fails = [&](int d) { return p(d, [&, d] { ++calls[d]; return false; }); };
  bool ok = works(0) && works(0) && calls[0] == 1;       // once on the first device
  ok = ok && !fails(1) && calls[1] == 1;                 // the second one's own result
  ok = ok && works(0) && calls[0] == 1;
  ok = ok && works(1) && calls[1] == 2 && works(1) && calls[1] == 2;  // a failure is not kept
  ok = ok && works(0) && !p(-1, [] { return false; }) && p(100000, [] { return true; });
  return ok ? 0 : 1;
}
"""


def test_each_device_is_set_up(tmp_path):
    (tmp_path / "t.cc").write_text(HARNESS)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-x", "c++", "-I", S.CSRC, str(tmp_path / "t.cc"), "-o", exe])
    assert subprocess.run([exe]).returncode == 0


@pytest.mark.parametrize("name", ["tree.cu", "forces.cu", "scan_sort.cu", "collide_spec.cu", "mlp.cu"])
def test_attributes_are_not_set_once_in_the_process(name):
    # (the set-up of a handle, in the other sources, runs with its device current)
    assert "cudaFuncSetAttribute" not in S.source(name)


@pytest.mark.parametrize("name, kernel", [
    ("tree.cu", "k_tree_small"), ("forces.cu", "k_link_block"), ("forces.cu", "k_mb_accumulate_block"),
    ("forces.cu", "k_mb_accumulate"), ("forces.cu", "k_mb_traverse_warp"), ("forces.cu", "k_mb_traverse"),
    ("scan_sort.cu", "k_sort_block"), ("noalloc.cu", "k_noalloc_out")])
def test_launches_are_checked(name, kernel):
    text = S.source(name)
    assert not re.search(r"D3_LAUNCH\(\(?%s[,<]" % kernel, text)
    assert re.search(r"\blaunch\(%s," % kernel, text)

"""Device buffers that are not to be had: room that only makes a pass faster
fails softly and is asked for less the next time, buffers that belong
together come all or not at all, and a size counts as held only when they
have come."""

import re
import subprocess

import pytest

import test_stream_order as S

HARNESS = r"""
#include <cstdlib>
#include <set>
#include "room.cuh"
using namespace d3;
// a device of `left` bytes
struct Device {
  size_t left;
  std::set<void *> held;
  size_t sizes = 0;
  bool take(void **p, size_t n) {
    if (n > left) return false;
    left -= n;
    *p = malloc(n + sizeof n);
    *(size_t *)*p = n;
    held.insert(*p);
    return true;
  }
  void give(void *p) {
    if (!p) return;
    if (!held.erase(p)) abort();  // given back twice
    left += *(size_t *)p;
    free(p);
  }
};
int main() {
  Device dev{1000};
  void *a = nullptr, *b = nullptr, *c = nullptr;
  auto take = [&](void **p, size_t n) { return dev.take(p, n); };
  auto give = [&](void *p) { dev.give(p); };
  auto three = [&](size_t n) { return take_all({{&a, n}, {&b, n}, {&c, n}}, take, give); };
  if (!three(300) || !a || !b || !c || dev.left != 100) return 1;
  for (void **p : {&a, &b, &c}) { give(*p); *p = nullptr; }
  if (three(400) || a || b || c || dev.left != 1000 || dev.held.size()) return 2;  // the third fails
  // spare room: nothing wanted, then more than there is, asked for in halves
  SpareRoom r{0, 0, 8192};
  int asked = 0;
  auto retake = [&](size_t n) {
    ++asked;
    for (void **p : {&a, &b, &c}) { give(*p); *p = nullptr; }
    return three(n);
  };
  r.grow(retake);
  if (asked || r.cap) return 3;
  r.want = 1000;
  uint32_t last = UINT32_MAX;
  for (int run = 0; run < 40; ++run) {
    r.grow(retake);
    if (r.cap == 0 && (dev.held.size() || r.limit >= last)) return 4;
    if (r.cap && dev.held.size() != 3) return 5;
    last = r.limit;
    if (r.cap) break;
  }
  if (r.cap < 156 || r.cap > 333) return 6;  // at least half of what fits
  const int before = asked;
  for (int run = 0; run < 5; ++run) r.grow(retake);
  if (asked != before) return 7;             // not asked for again on every run
  // no room at all: given up after a bounded number of tries
  Device none{0};
  dev = none;
  a = b = c = nullptr;
  SpareRoom q{0, 5000, 8192};
  asked = 0;
  for (int run = 0; run < 100; ++run) q.grow(retake);
  if (q.cap || asked > 14) return 8;
  // grows with what is wanted, by a quarter more, up to the limit
  dev.left = 1 << 20;
  SpareRoom g{0, 100, 8192};
  g.grow(retake);
  if (g.cap != 125) return 9;
  g.want = 126;
  g.grow(retake);
  g.want = 1000000;
  g.grow(retake);
  return g.cap == 8192 ? 0 : 10;
}
"""


def test_room_policy(tmp_path):
    (tmp_path / "t.cc").write_text(HARNESS)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-x", "c++", "-I", S.CSRC, str(tmp_path / "t.cc"), "-o", exe])
    assert subprocess.run([exe]).returncode == 0


def test_long_lists_go_without_their_room():
    text = S.function("fmm_run", S.source("fmm.cu"))
    assert not re.search(r"D3_CUDA_OK\(cudaMalloc\(&f\.long", text)
    assert "long_room.grow(" in text


def test_segments_go_without_their_room():
    text = S.source("fmm_tc.cu")
    assert "device_take" in S.function("segment_sums", text) and "grow_parts" not in text
    # a kernel that could meet a split list asks whether there is room for its sums
    for kernel in ("k_tc_near", "k_tc_far"):
        for use in re.findall(r"[^;]*\bmore_segments\(", S.function(kernel, text)):
            assert re.search(r"a\.part_(p2p|w) (&&|\?)", use), use


@pytest.mark.parametrize("name, function", [
    ("fmm.cu", "fmm_run"), ("fmm.cu", "fmm_reserve_points"), ("fmm.cu", "fmm_reserve_cells"),
    ("fmm_tc.cu", "reserve"), ("fmm_tc.cu", "tc_run")])
def test_a_size_is_held_when_its_buffers_have_come(name, function):
    # each group: its size to 0, the old buffers back, all the new ones or a
    # return, then the size
    text = S.function(function, S.source(name))
    assert not re.search(r"\bcudaMalloc\(", text)
    groups = re.findall(r"(\w)\.(\w*cap) = 0;\s*device_give\(([^)]*)\);(.*?)\1\.\2 = (?!0)", text, re.S)
    assert len(groups) == len(re.findall(r"\bdevice_give\(", text)) - text.count(".grow([&]")
    for _, _, given, between in groups:
        taken = re.findall(r"\(void \*\*\)&(\w\.\w+)", between)
        assert taken == [p.strip() for p in given.split(",")]
        assert "return -1;" in between

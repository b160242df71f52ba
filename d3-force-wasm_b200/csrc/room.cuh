// room.cuh - device buffers that may not be to be had (plain C++, so that a
// host test can compile it).
#pragma once

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace d3 {

// A buffer to take: the pointer (null until then) and its bytes.
struct Want {
  void **p;
  size_t bytes;
};

// All of the buffers, or none: false, every pointer null again. take(p, bytes)
// sets *p (true) or leaves it; give(p) frees.
template <class Take, class Give>
bool take_all(std::initializer_list<Want> wants, Take take, Give give) {
  for (const Want &w : wants) {
    if (take(w.p, w.bytes)) continue;
    for (const Want &u : wants) {
      give(*u.p);
      *u.p = nullptr;
    }
    return false;
  }
  return true;
}

// Room that only makes a pass faster: grown to what a run wanted and a quarter
// more, where that is to be had. Where it is not, the pass goes without, and
// the next one that wants more asks for half as much at most.
struct SpareRoom {
  uint32_t cap = 0, want = 0, limit = UINT32_MAX;

  // retake(units): the old buffers go, new ones of `units` come (true) or none
  template <class Retake>
  void grow(Retake retake) {
    if (want <= cap || cap >= limit) return;
    const uint64_t roomy = (uint64_t)want + want / 4;
    const uint32_t units = roomy < limit ? (uint32_t)roomy : limit;
    if (retake(units)) {
      cap = units;
    } else {
      cap = 0;
      limit = units / 2;
    }
  }
};

}  // namespace d3

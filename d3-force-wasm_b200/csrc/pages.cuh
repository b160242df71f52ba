// pages.cuh - which of a buffer's pages have memory behind them (plain C++, so
// that a host test can compile it).
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>

namespace d3 {

// About how many bytes of [p, p + bytes) were never touched (a write to them
// takes a page fault), from `samples` pages spread over it. Where the kernel
// does not say, none.
inline size_t untouched_bytes(const void *p, size_t bytes, unsigned samples = 16) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  const uintptr_t first = ((uintptr_t)p + page - 1) / page * page, end = ((uintptr_t)p + bytes) / page * page;
  if (end <= first) return 0;
  const size_t pages = (end - first) / page;
  const size_t looks = pages < samples ? pages : samples;
  size_t untouched = 0;
  for (size_t k = 0; k < looks; ++k) {
    unsigned char in = 1;
    void *at = reinterpret_cast<void *>(first + (pages * (2 * k + 1) / (2 * looks)) * page);
    if (mincore(at, page, &in) == 0 && !(in & 1)) ++untouched;
  }
  return (size_t)((double)bytes * untouched / looks);
}

}  // namespace d3

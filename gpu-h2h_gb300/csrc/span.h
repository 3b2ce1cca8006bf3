// span.h -- whether a kernel may read a caller's ints in place.
#pragma once

#include <cstdint>

namespace gh {

// The n ints at address p lie within the `size` bytes at `start` and are
// aligned as the device reads them.
inline bool ints_inside(uint64_t p, int64_t n, uint64_t start, uint64_t size) {
  return p % sizeof(int) == 0 && p >= start && p - start <= size && n >= 0 &&
         (uint64_t)n <= (size - (p - start)) / sizeof(int);
}

}  // namespace gh

// arena.h -- device arrays of one phase or object, cut from a few allocations
// and freed together.  cudaMalloc and cudaFree of a small array cost about 60
// us a pair (the free waits for the device); a build makes some 150 arrays, so
// on a 4,096-vertex graph they were half of its time.
#pragma once

#include <algorithm>
#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include "common.h"

namespace gh {

// One allocation of n elements.  Without room the CUDA error is cleared before
// the exception leaves, so that no later check trips over it.
template <typename T>
T *device_array(int64_t n) {
  void *p = nullptr;
  const cudaError_t e = cudaMalloc(&p, (size_t)std::max<int64_t>(n, 1) * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error(H2H_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  return static_cast<T *>(p);
}

class DeviceArena {
 public:
  DeviceArena() = default;
  DeviceArena(const DeviceArena &) = delete;
  DeviceArena &operator=(const DeviceArena &) = delete;
  ~DeviceArena() { release(); }

  // Room for arrays of `total` bytes in all (each rounded up to 256) in one
  // allocation, for a phase that knows what it will take.
  void reserve(size_t total) {
    cur_ = chunk(total);
    cap_ = total;
    used_ = 0;
  }

  // n elements, aligned to 256 bytes, uninitialised.  What the current chunk
  // has no room for and takes 8 MiB or more is an allocation of its own; smaller
  // arrays share chunks that double up to 64 MiB.
  template <typename T>
  T *get(int64_t n) {
    const size_t want = ((size_t)std::max<int64_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
    bytes += (int64_t)((size_t)std::max<int64_t>(n, 1) * sizeof(T));
    if (want > cap_ - used_) {
      if (want >= (size_t(8) << 20)) return reinterpret_cast<T *>(chunk(want));
      next_ = std::min<size_t>(std::max<size_t>(2 * next_, size_t(1) << 20), size_t(64) << 20);
      const size_t size = std::max(want, next_);
      cur_ = chunk(size);
      cap_ = size;
      used_ = 0;
    }
    char *p = cur_ + used_;
    used_ += want;
    return reinterpret_cast<T *>(p);
  }

  // Frees everything (waits for the device, as cudaFree does).
  void release() {
    for (void *p : chunks_) cudaFree(p);
    chunks_.clear();
    cur_ = nullptr;
    cap_ = used_ = next_ = 0;
    bytes = 0;
  }

  int64_t bytes = 0;  // of the arrays handed out

 private:
  char *chunk(size_t size) {
    char *p = device_array<char>((int64_t)size);
    chunks_.push_back(p);
    return p;
  }
  std::vector<void *> chunks_;
  char *cur_ = nullptr;
  size_t cap_ = 0, used_ = 0, next_ = 0;
};

}  // namespace gh

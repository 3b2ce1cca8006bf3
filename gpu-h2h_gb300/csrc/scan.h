// scan.h -- exclusive prefix sums on the GPU and the scratch memory they take,
// shared by the loader, the elimination sets, the tree build and the label
// fill's plan.
#pragma once

#include <algorithm>
#include <cstdint>

#include "arena.h"

namespace gh {

namespace {

constexpr int kScanThreads = 1024, kScanItems = 4, kScanTile = kScanThreads * kScanItems;

template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(const T *in, int64_t *out, int64_t n,
                                                                 int64_t *tile_sums) {
  __shared__ int64_t warp_tot[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)tid * kScanItems;
  int64_t v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    v[k] = base + k < n ? (int64_t)in[base + k] : 0;
    s += v[k];
  }
  int64_t x = s;  // inclusive warp scan of the thread sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int64_t t = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    warp_tot[lane] = t;  // inclusive over warps
  }
  __syncthreads();
  int64_t run = x - s + (wid > 0 ? warp_tot[wid - 1] : 0);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (tid == kScanThreads - 1) tile_sums[blockIdx.x] = run;
}

__global__ void scan_add_kernel(int64_t *out, int64_t n, const int64_t *tile_offsets) {
  const int64_t add = tile_offsets[blockIdx.x];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  for (int i = threadIdx.x; i < kScanTile; i += blockDim.x)
    if (base + i < n) out[base + i] += add;
}

// Device scratch of one build, freed together.
using Workspace = DeviceArena;

// out[i] = sum of in[0 .. i) for i < n (tile sums scanned recursively).
template <typename T>
void exclusive_scan(const T *in, int64_t *out, int64_t n, Workspace &ws, cudaStream_t s) {
  if (n <= 0) return;
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  int64_t *sums = ws.get<int64_t>(tiles);
  scan_tile_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, sums);
  GH_CUDA(cudaGetLastError());
  if (tiles > 1) {
    int64_t *offs = ws.get<int64_t>(tiles);
    exclusive_scan<int64_t>(sums, offs, tiles, ws, s);
    scan_add_kernel<<<(unsigned)tiles, 256, 0, s>>>(out, n, offs);
    GH_CUDA(cudaGetLastError());
  }
}

}  // namespace

}  // namespace gh

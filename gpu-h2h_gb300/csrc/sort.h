// sort.h -- a stable radix sort of (key, value) pairs on the GPU, shared by the
// loader (input_gpu.cu) and the tree build (tree_gpu.cu).
#pragma once

#include "scan.h"

namespace gh {

namespace {

// Stable LSD radix sort of (uint32 key, int32 value) pairs, 8 bits a pass.
// A tile of 4,096 pairs is 8 warps x 16 rounds of 32 consecutive pairs; a
// pair's place in its digit's run is the digit's global offset for the tile
// (a scan over digit-major tile histograms) plus the pairs of that digit
// before it in the tile, counted warp by warp and round by round with
// __match_any_sync, so equal digits keep their input order.

constexpr int kRadixThreads = 256, kRadixRounds = 16, kRadixTile = kRadixThreads * kRadixRounds, kBins = 256;

__global__ void __launch_bounds__(kRadixThreads) radix_hist_kernel(const unsigned *keys, int64_t n, int shift,
                                                                   int *hist, int ntiles) {
  __shared__ int cnt[kBins];
  for (int b = threadIdx.x; b < kBins; b += blockDim.x) cnt[b] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRadixTile;
  for (int i = threadIdx.x; i < kRadixTile; i += blockDim.x)
    if (base + i < n) atomicAdd(&cnt[(keys[base + i] >> shift) & (kBins - 1)], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < kBins; b += blockDim.x) hist[(int64_t)b * ntiles + blockIdx.x] = cnt[b];
}

__global__ void __launch_bounds__(kRadixThreads) radix_scatter_kernel(const unsigned *kin, const int *vin,
                                                                      unsigned *kout, int *vout, int64_t n, int shift,
                                                                      const int64_t *offs, int ntiles) {
  __shared__ int64_t wpos[kRadixThreads / 32][kBins];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int b = lane; b < kBins; b += 32) wpos[w][b] = 0;
  __syncwarp();
  const int64_t wbase = (int64_t)blockIdx.x * kRadixTile + (int64_t)w * 32 * kRadixRounds;
  const unsigned lt = (1u << lane) - 1;
  for (int r = 0; r < kRadixRounds; r++) {  // per-warp digit counts
    const int64_t i = wbase + r * 32 + lane;
    const bool valid = i < n;
    const unsigned d = valid ? (kin[i] >> shift) & (kBins - 1) : kBins;
    const unsigned mask = __match_any_sync(0xffffffffu, d);
    if (valid && (mask & lt) == 0) wpos[w][d] += __popc(mask);
    __syncwarp();
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kBins; b += blockDim.x) {  // warp starts inside the digit's run
    int64_t run = offs[(int64_t)b * ntiles + blockIdx.x];
    for (int ww = 0; ww < kRadixThreads / 32; ww++) {
      const int64_t c = wpos[ww][b];
      wpos[ww][b] = run;
      run += c;
    }
  }
  __syncthreads();
  for (int r = 0; r < kRadixRounds; r++) {
    const int64_t i = wbase + r * 32 + lane;
    const bool valid = i < n;
    const unsigned key = valid ? kin[i] : 0u;
    const unsigned d = valid ? (key >> shift) & (kBins - 1) : kBins;
    const unsigned mask = __match_any_sync(0xffffffffu, d);
    if (valid) {
      const int64_t pos = wpos[w][d] + __popc(mask & lt);
      if (pos >= 0 && pos < n) {
        kout[pos] = key;
        vout[pos] = vin[i];
      }
    }
    __syncwarp();
    if (valid && (mask & lt) == 0) wpos[w][d] += __popc(mask);
    __syncwarp();
  }
}

// Sorts keys/vals (n pairs, keys < 2^bits) stably by key; the result is in
// keys/vals.
void radix_sort_pairs(unsigned *keys, int *vals, int64_t n, int bits, Workspace &ws, cudaStream_t s) {
  if (n <= 1) return;
  const int ntiles = (int)((n + kRadixTile - 1) / kRadixTile);
  unsigned *k2 = ws.get<unsigned>(n);
  int *v2 = ws.get<int>(n);
  int *hist = ws.get<int>((int64_t)kBins * ntiles);
  int64_t *offs = ws.get<int64_t>((int64_t)kBins * ntiles);
  unsigned *ka = keys, *kb = k2;
  int *va = vals, *vb = v2;
  for (int shift = 0; shift < bits; shift += 8) {
    radix_hist_kernel<<<ntiles, kRadixThreads, 0, s>>>(ka, n, shift, hist, ntiles);
    GH_CUDA(cudaGetLastError());
    exclusive_scan<int>(hist, offs, (int64_t)kBins * ntiles, ws, s);
    radix_scatter_kernel<<<ntiles, kRadixThreads, 0, s>>>(ka, va, kb, vb, n, shift, offs, ntiles);
    GH_CUDA(cudaGetLastError());
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    GH_CUDA(cudaMemcpyAsync(keys, ka, sizeof(unsigned) * n, cudaMemcpyDeviceToDevice, s));
    GH_CUDA(cudaMemcpyAsync(vals, va, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  }
}

int bits_for(int64_t maxval) {
  int b = 1;
  while (b < 32 && (int64_t(1) << b) <= maxval) b++;
  return b;
}

}  // namespace

}  // namespace gh

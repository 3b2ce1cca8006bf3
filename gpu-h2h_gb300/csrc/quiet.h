// quiet.h -- device work of calls that are plain host calls to their caller
// (loading, reading a graph or its tree back).
#pragma once

#include "common.h"

namespace gh {

namespace {

// The caller, or another thread of the program, may be capturing a graph: allocations
// must not count against the capture, and no work goes to the legacy stream.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  RelaxedCapture(const RelaxedCapture &) = delete;
  RelaxedCapture &operator=(const RelaxedCapture &) = delete;
};

// The calling thread's device for a while.
struct OnDevice {
  int before = 0;
  explicit OnDevice(int device) {
    GH_CUDA(cudaGetDevice(&before));
    if (device != before) GH_CUDA(cudaSetDevice(device));
  }
  ~OnDevice() { cudaSetDevice(before); }
  OnDevice(const OnDevice &) = delete;
  OnDevice &operator=(const OnDevice &) = delete;
};

struct QuietStream {
  cudaStream_t s = nullptr;
  QuietStream() { GH_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
  ~QuietStream() {
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
  }
  QuietStream(const QuietStream &) = delete;
  QuietStream &operator=(const QuietStream &) = delete;
  void read(void *to, const void *from, size_t bytes) {
    GH_CUDA(cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToHost, s));
    GH_CUDA(cudaStreamSynchronize(s));
  }
};

}  // namespace

}  // namespace gh

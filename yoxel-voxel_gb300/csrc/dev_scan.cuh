// dev_scan.cuh - device helpers shared by the scene builders: stream-ordered
// scratch buffers and grid sizing.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "yv_kernels.h"

namespace yv {
namespace {

// Device buffers released on scope exit (stream-ordered).
struct DevBuf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  cudaError_t alloc(size_t bytes, cudaStream_t st) {
    s = st;
    return scratch_alloc(&p, bytes ? bytes : 16, st);
  }
  ~DevBuf() { scratch_free(p, s); }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

int grid_for(uint64_t work) {
  const uint64_t b = (work + 255) / 256;
  const uint64_t cap = (uint64_t)device_sm_count() * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace
}  // namespace yv

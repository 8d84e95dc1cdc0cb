// zg_scratch.cuh — scratch of one call from the library's pool (zg_malloc_async), given back on the
// call's stream.  A cudaMalloc/cudaFree pair costs 50-200 us and synchronises the device; a graph
// build needs ten of them.
#pragma once

#include "zg_internal.cuh"

struct ZgScratch {
  void* p = nullptr;
  cudaStream_t s;
  explicit ZgScratch(cudaStream_t stream) : s(stream) {}
  ZgScratch(const ZgScratch&) = delete;
  ZgScratch& operator=(const ZgScratch&) = delete;
  ~ZgScratch() { reset(); }
  int alloc(size_t bytes) {
    reset();
    cudaError_t e = zg_malloc_async(&p, bytes ? bytes : 1, s);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      zg_trim_pool(s);
      e = zg_malloc_async(&p, bytes ? bytes : 1, s);
    }
    if (e == cudaSuccess) return ZG_OK;
    cudaGetLastError();
    p = nullptr;
    const int code = e == cudaErrorMemoryAllocation ? ZG_ERR_OOM : ZG_ERR_CUDA;
    zg_set_error(code, "scratch of %zu bytes: %s", bytes, cudaGetErrorString(e));
    return code;
  }
  void reset() {
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
  }
  template <typename T>
  T* as(size_t at = 0) const {
    return (T*)((char*)p + at);
  }
};

// Offsets of several arrays in one allocation.
struct ZgCarve {
  size_t at = 0;
  size_t take(size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) & ~(size_t)255;
    return p;
  }
};

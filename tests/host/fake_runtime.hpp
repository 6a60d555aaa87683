// Stand-ins for the CUDA runtime calls of the library's host code: "device" memory is host memory,
// streams run at once, and a test can make the next calls of a kind fail. Included by one
// translation unit of a test program.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace fake {
struct Call {
  std::atomic<int> calls{0}, fail{0};  // fail: calls that still return an error
  cudaError_t run() {
    ++calls;
    int f = fail.load();
    while (f > 0 && !fail.compare_exchange_weak(f, f - 1)) {
    }
    return f > 0 ? cudaErrorMemoryAllocation : cudaSuccess;
  }
};
inline Call malloc_, memset_;
}  // namespace fake

#define CHECK(cond)                                              \
  do {                                                           \
    if (!(cond)) {                                               \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #cond);    \
      std::exit(1);                                              \
    }                                                            \
  } while (0)

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  const cudaError_t e = fake::malloc_.run();
  if (e == cudaSuccess) {
    *p = std::malloc(n);
    std::memset(*p, 0xAB, n);  // device memory starts as anything but zero
  }
  return e;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  const cudaError_t e = fake::memset_.run();
  if (e == cudaSuccess) std::memset(p, v, n);
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
}

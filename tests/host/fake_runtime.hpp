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
    if (f > 0) left();
    return f > 0 ? cudaErrorMemoryAllocation : cudaSuccess;
  }
  static void left();
};
inline Call malloc_, memset_, host_alloc, host_free, stream_create, copy;
inline std::atomic<int> streams{0};
inline std::atomic<bool> error_left{false};   // a failed call's code not yet taken by cudaGetLastError
inline const char *pinned_from = nullptr, *pinned_to = nullptr;  // memory the test declares pinned
inline void Call::left() { error_left = true; }
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
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  const cudaError_t e = fake::host_alloc.run();
  if (e == cudaSuccess) *p = std::malloc(n);
  return e;
}
cudaError_t cudaFreeHost(void* p) {
  fake::host_free.run();
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  const cudaError_t e = fake::stream_create.run();
  if (e == cudaSuccess) *s = (cudaStream_t)(size_t)++fake::streams;
  return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  const cudaError_t e = fake::copy.run();
  if (e == cudaSuccess) std::memcpy(d, s, n);
  return e;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = (const char*)p >= fake::pinned_from && (const char*)p < fake::pinned_to ? cudaMemoryTypeHost
                                                                                   : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  return fake::error_left.exchange(false) ? cudaErrorMemoryAllocation : cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
}

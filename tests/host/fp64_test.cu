// The device functions of csrc/fp64.hpp, one thread an element, for tests/test_gpu_fp64.py.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../pcaone_b200/csrc/fp64.hpp"

namespace {
__global__ void evaluate(int op, int64_t n, const double* a, const double* b, double* out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  out[i] = op == 0   ? pg::fast_reciprocal(x)
           : op == 1 ? pg::reciprocal(x)
           : op == 2 ? pg::quotient(y, x, pg::reciprocal(x))
                     : y / x;
}
}  // namespace

extern "C" int fp64_evaluate(int op, int64_t n, const double* a, const double* b, double* out) {
  double *d = nullptr;
  cudaError_t e = cudaMalloc(&d, 3 * n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    evaluate<<<(unsigned)((n + 255) / 256), 256>>>(op, n, d, d + n, d + 2 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}

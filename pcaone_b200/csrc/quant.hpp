// Fixed-point pieces of the int8 decode-GEMM's sketch operand (kernels_gemm_i8.cu): the layout
// and the rounding, shared by the kernels that write it.
#pragma once

#include <cstdint>

namespace pg {

constexpr int kI8Chunk = 128;  // operand rows per K chunk

// Column layout: piece p of column c is row p * LP + c of the chunk's image (and column
// p * LP + c of the accumulator), LP = l rounded up to 8; NP rows of 128 bytes in all.
__host__ __device__ constexpr int i8_lp(int l) { return (l + 7) / 8 * 8; }
__host__ __device__ constexpr int i8_np(int l) { return (3 * i8_lp(l) + 15) / 16 * 16; }

// Piece scales of a column from its maximum (the bits of a double): sig0 = max / 127,
// sig1 = sig0 / 254, sig2 = sig1 / 254, in FP32 (the same values in the quantiser and in the
// GEMM readout).
__device__ __forceinline__ void piece_scales(unsigned long long bits, float* s) {
  const double mx = __longlong_as_double((long long)bits);
  s[0] = mx > 0.0 ? (float)(mx / 127.0) : 1.0f;
  s[1] = s[0] / 254.0f;
  s[2] = s[1] / 254.0f;
}

// Scales (and their reciprocals, one division a column instead of three an element) of the lp
// columns of a chunk image in shared memory; `write` also stores the 3 x lp scales to sig.
struct PieceTable {
  double s[3][64], inv[3][64];
  __device__ __forceinline__ void fill(const unsigned long long* qmax, int l, int lp, float* sig, bool write) {
    for (int c = threadIdx.x; c < lp; c += blockDim.x) {
      float f[3] = {1.0f, 1.0f, 1.0f};
      if (c < l) piece_scales(qmax[c], f);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        s[p][c] = (double)f[p];
        inv[p][c] = 1.0 / (double)f[p];
        if (write) sig[p * lp + c] = f[p];
      }
    }
  }
  // The three pieces of element (row kk of the chunk, column c), each the rounded residual of the
  // previous ones (|q| <= 127), into the image img (NP rows of 128 bytes): byte
  // 8 (o & 1) + (o >> 1) of 16-byte unit u for u = kk / 16, o = kk % 16 (the decoder's code
  // order), units 128-byte swizzled.
  __device__ __forceinline__ void put(uint8_t* img, int kk, int c, int lp, double x) const {
    const int u = kk >> 4, o = kk & 15, pp = 8 * (o & 1) + (o >> 1);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const double q = fmin(127.0, fmax(-127.0, rint(x * inv[p][c])));
      x -= q * s[p][c];
      const int n = p * lp + c;
      img[n * 128 + ((u ^ (n & 7)) << 4) + pp] = (uint8_t)(int8_t)(int)q;
    }
  }
};

}  // namespace pg

// Fused Omega update (kernels_update.cu).
#pragma once

#include <cuda_bf16.h>

#include "internal.hpp"

namespace pg {

// The int8 back end's operand copy of Omega (kernels_gemm_i8.cu): column maxima (bits of
// doubles), the chunked pieces (kpad / 128 chunk images) and their scales.
struct OmegaI8 {
  unsigned long long* qmax = nullptr;
  int8_t* bq = nullptr;
  float* sig = nullptr;
};

struct UpdateArgs {
  double* H1 = nullptr;        // the sketch is H1 + H2 (written to H) when H2 is given, else H
  const double* H2 = nullptr;
  double* H = nullptr;
  double* Q = nullptr;         // N x l work: the orthonormal factor before the signs
  double* Omg = nullptr;       // N x l: the previous Omega in, the new one out
  float* Omgf = nullptr;       // FP32 operand copy (SIMT path) or null
  OmegaI8 i8;                  // int8 operand (bq null: none)
  __nv_bfloat16* bt1 = nullptr;  // split-BF16 operand (tc_layout.hpp) or null
  int bt_half = 0;               // row offset of the lo half in bt1 (= NP / 2)
  int64_t kpad = 0;            // padded rows of the operand copies (a multiple of 128)
  double* wsum = nullptr;      // l column sums of the new Omega
  double* D = nullptr;         // l
  double* mult = nullptr;      // l
  double *R1i = nullptr, *R2i = nullptr;  // l x l work
  int* status = nullptr;
  int64_t N = 0;
  int l = 0;
  // set by fused_update
  double* part = nullptr;
  unsigned* counter = nullptr;
};

void fused_update(pcaone_ctx* c, UpdateArgs a);

}  // namespace pg

// FP64 linear algebra on tall row-major matrices (n x l, l <= kLmax): kernels_linalg.cu.
#pragma once

#include "internal.hpp"

namespace pg {

// One pass over the rows of A and what the CTA that finishes last makes of the result.
//   rows:  x = A (+ A2, stored to Asum; without Rinv only);  q = x Rinv when Rinv is given (stored
//          to Q, which may be A itself unless B is given), else x
//   Gram (B null):  W = q^T q = R^T R:  R, Ri = R^-1; with Rprev also Racc = R Rprev and, with
//          Rprev_inv = Rprev^-1, Racc_inv = Rprev_inv Ri. status[0] gets 1 + the first column
//          whose pivot is not positive.
//   cross (B, n x lb, lb <= l; needs Rinv):  X (l x lb) = q^T B; Ri, R, ... unused
// Square factors are l x l row-major, upper with zeros below; null outputs are not written.
struct TallStep {
  const double* A = nullptr;
  const double* A2 = nullptr;
  double* Asum = nullptr;
  const double* Rinv = nullptr;
  double* Q = nullptr;
  const double* B = nullptr;
  int lb = 0;
  double* X = nullptr;
  double *R = nullptr, *Ri = nullptr;
  const double *Rprev = nullptr, *Rprev_inv = nullptr;
  double *Racc = nullptr, *Racc_inv = nullptr;
  int* status = nullptr;
  int64_t n = 0;
  int l = 0;
  // set by tall_step
  double* part = nullptr;
  unsigned* counter = nullptr;
};
void tall_step(pcaone_ctx* c, TallStep s);
// Ticket counter of the tall kernels (zero between launches; buffers.cu) and room for the sums of
// kTallMaxParts clusters of up to `doubles` each.
unsigned* tall_counter(pcaone_ctx* c);
double* tall_part(pcaone_ctx* c, size_t doubles);

// Q = A R^-1 (may alias A == Q).
void trsm_right_upper(pcaone_ctx* c, const double* A, const double* R, int l, int64_t n, double* Q);
void colsum(pcaone_ctx* c, const double* A, int l, int64_t n, double* out);
// Y (n x kc) = X (n x l) * C[:, :kc] with C l x ldc row-major.
void rowmat(pcaone_ctx* c, const double* X, int l, const double* C, int ldc, int kc, int64_t n, double* Y);

// Column-major n x l (the hosts' layout) -> row-major npad x l, zero past row n, column j scaled by
// scale[j] when scale (device) is given, and an optional FP32 copy; and back (row stride ld).
void to_rowmajor(pcaone_ctx* c, const double* cm, int64_t n, int l, int64_t npad, const double* scale, double* out,
                 float* outf = nullptr);
void to_colmajor(pcaone_ctx* c, const double* X, int64_t n, int l, int ld, double* out);

}  // namespace pg

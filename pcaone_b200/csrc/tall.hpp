// Building blocks of the FP64 kernels on tall row-major matrices (n rows, l <= 64 columns):
// Gram products, products with a small upper factor, and the l x l factorisations that one CTA
// does between them.
//
// All of it runs on the FP64 tensor-core shape m8n8k4 (36 TFLOP/s measured here from eight warps
// an SM on, against 28-34 for FMA chains), chosen for its operand layout rather than its rate:
// a warp's operand of 4 rows x 8 columns (lane: row lane % 4, column lane / 4) is the same
// register for A^T and for A, so the Gram of 4 rows needs one 8-byte load a lane and column
// tile, straight from global memory, and no shared memory. A product Q = X Rinv computed
// transposed (Rinv^T X^T) leaves its 8 x 8 result in exactly that layout (rows 0, 2, 4, 6 in
// the lane's first register, 1, 3, 5, 7 in the second), so Q feeds the Gram from registers.
//
// Reductions run in a fixed order (warps of the CTA, CTAs of the cluster through distributed
// shared memory, clusters by the CTA that finishes last), so results are deterministic.
#pragma once

#include <cooperative_groups.h>

#include "fp64.hpp"
#include "internal.hpp"

namespace pg {

namespace cg = cooperative_groups;

constexpr int kTallThreads = 256;  // 8 warps; a warp takes 8 rows at a time
constexpr int kTallWarps = kTallThreads / 32;
constexpr int kTallCluster = 8;    // CTAs per cluster
constexpr int kTallMaxParts = 36;  // clusters of a launch: the last CTA reads one sum of each

// d (8x8) += a (8x4) b (4x8): lane holds a[lane/4][lane%4], b[lane%4][lane/4] and
// d[lane/4][2 (lane%4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// NT column tiles of 8: padded width and the row stride of l x l matrices in shared memory (the
// stride 4 mod 16 makes the 4 x 4 element reads of a half warp conflict-free).
template <int NT>
struct Tall {
  static constexpr int LT = 8 * NT, LD = LT + 4;
  static constexpr int kTiles = NT * (NT + 1) / 2;    // tiles on and above the diagonal
  static constexpr int kSq = LT * LD;                 // doubles of an l x l matrix
  static constexpr int kWarpScratch = 256 + kTallWarps * 64;  // 8 x 8 blocks of the factorisations
  static __device__ __forceinline__ constexpr int tile(int i, int j) { return i * NT - i * (i - 1) / 2 + (j - i); }
};

// Rows per CTA when at most `ctas` CTAs split n rows: a multiple of 64, so that every warp takes
// the same number of 8-row groups.
__host__ __device__ __forceinline__ int64_t tall_rows_per_cta(int64_t n, int64_t ctas) {
  return ((n + ctas - 1) / ctas + 63) & ~int64_t(63);
}
// Clusters for n rows, at most cap of them (one where the device holds no more at once: what a
// launch sets aside for other work may leave cap at 0).
inline int tall_clusters(int64_t n, int cap) {
  if (cap < 1) cap = 1;
  const int64_t per = kTallCluster * tall_rows_per_cta(n, (int64_t)cap * kTallCluster);
  return (int)((n + per - 1) / per);
}
// Row range of CTA `cta` of `ctas`.
__device__ __forceinline__ void tall_rows(int64_t n, int64_t cta, int64_t ctas, int64_t& r0, int64_t& r1) {
  const int64_t rpb = tall_rows_per_cta(n, ctas);
  r0 = cta * rpb < n ? cta * rpb : n;
  r1 = r0 + rpb < n ? r0 + rpb : n;
}

// Copy the l x l row-major matrix src into shared memory (row stride LD); `diag` on the padded
// diagonal, zeros elsewhere.
template <int NT>
__device__ __forceinline__ void load_square(const double* src, int l, double diag, double* dst) {
  for (int t = threadIdx.x; t < Tall<NT>::LT * Tall<NT>::LT; t += blockDim.x) {
    const int i = t / Tall<NT>::LT, j = t - i * Tall<NT>::LT;
    dst[i * Tall<NT>::LD + j] = (i < l && j < l) ? src[i * l + j] : (i == j ? diag : 0.0);
  }
}

template <int NT>
__device__ __forceinline__ void store_square(const double* src, int l, double* dst) {
  for (int t = threadIdx.x; t < l * l; t += blockDim.x) dst[t] = src[(t / l) * Tall<NT>::LD + t % l];
}

// d += op(A) B for 8 x 8 blocks in shared memory (row strides lda, ldb); op(A) = A^T when TA.
template <bool TA>
__device__ __forceinline__ void block_mma(double (&d)[2], const double* A, int lda, const double* B, int ldb,
                                          double sign = 1.0) {
  const int q = (threadIdx.x & 31) >> 2, r = threadIdx.x & 3;
#pragma unroll
  for (int h = 0; h < 8; h += 4)
    dmma(d, sign * (TA ? A[(h + r) * lda + q] : A[q * lda + h + r]), B[(h + r) * ldb + q]);
}
__device__ __forceinline__ void block_load(double (&d)[2], const double* C, int ldc) {
  const int q = (threadIdx.x & 31) >> 2, r = threadIdx.x & 3;
  const double2 v = *reinterpret_cast<const double2*>(C + q * ldc + 2 * r);
  d[0] = v.x;
  d[1] = v.y;
}
__device__ __forceinline__ void block_store(const double (&d)[2], double* C, int ldc) {
  const int q = (threadIdx.x & 31) >> 2, r = threadIdx.x & 3;
  *reinterpret_cast<double2*>(C + q * ldc + 2 * r) = make_double2(d[0], d[1]);
}

// The 8 x 8 block factorisations run in one warp, lane (g, r) = (lane / 8, lane % 8) holding row r,
// columns 2 g and 2 g + 1, so that a step is the same few instructions for every column: the code
// runs once a launch, on a CTA whose SM has not fetched it, and unrolled over the columns of a
// row a lane it cost more in instruction fetches than in arithmetic.

// Cholesky factor R_bb of the symmetric block Wb (row stride LD) into Rb and its inverse into Xb
// (upper, zeros below), and the inverse of R_bb^T into Li (8 x 8). A step eliminates one column of
// the block and of an identity beside it, which ends as the inverse of the unit lower factor;
// the square roots of the pivots are taken at once at the end. A pivot that is not positive, normal
// and finite is replaced by 1: returns 1 + the first one's index, else 0.
template <int LD>
__device__ __forceinline__ int chol_block(const double* Wb, double* Rb, double* Xb, double* Li) {
  const int lane = threadIdx.x & 31, r = lane & 7, g = lane >> 3, row0 = lane & 24;
  double d0 = Wb[r * LD + 2 * g], d1 = Wb[r * LD + 2 * g + 1], own = 1.0;
  double y0 = r == 2 * g ? 1.0 : 0.0, y1 = r == 2 * g + 1 ? 1.0 : 0.0;
  int bad = 0;
#pragma unroll 1
  for (int jj = 0; jj < 4; ++jj)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 2 * jj + h;
      const double dj = h ? d1 : d0;
      double p = __shfl_sync(0xffffffffu, dj, 8 * jj + j);
      const double m = __shfl_sync(0xffffffffu, dj, 8 * jj + r);
      const double w0 = __shfl_sync(0xffffffffu, d0, row0 + j), w1 = __shfl_sync(0xffffffffu, d1, row0 + j);
      const double v0 = __shfl_sync(0xffffffffu, y0, row0 + j), v1 = __shfl_sync(0xffffffffu, y1, row0 + j);
      if (!(p >= 2.3e-308 && p < 4e307)) {
        if (!bad) bad = j + 1;
        p = 1.0;
      }
      if (r == j) own = p;
      const double f = r > j ? m * fast_reciprocal(p) : 0.0;
      d0 = 2 * g > j ? d0 - f * w0 : 2 * g == j ? f : d0;
      d1 = 2 * g + 1 > j ? d1 - f * w1 : 2 * g + 1 == j ? f : d1;
      y0 -= f * v0;
      y1 -= f * v1;
    }
  const double iroot = rsqrt(own), root = own * iroot;
  const double s0 = __shfl_sync(0xffffffffu, root, 2 * g), s1 = __shfl_sync(0xffffffffu, root, 2 * g + 1);
  Rb[2 * g * LD + r] = r == 2 * g ? s0 : d0 * s0;
  Rb[(2 * g + 1) * LD + r] = r == 2 * g + 1 ? s1 : d1 * s1;
  Xb[2 * g * LD + r] = Li[r * 8 + 2 * g] = y0 * iroot;
  Xb[(2 * g + 1) * LD + r] = Li[r * 8 + 2 * g + 1] = y1 * iroot;
  __syncwarp();
  return bad;
}

// Cholesky W = R^T R of the l x l matrix in shared memory (tiles on and above the diagonal read,
// W overwritten; padded to LT with a unit diagonal) and X = R^-1, both upper with zeros below.
// Blocks of 8: warp 0 factors and inverts the diagonal block (chol_block, 8 steps in registers),
// the block row and the trailing tiles are block products spread over the warps, and warp 0 goes
// on from the next diagonal tile to its factor while the others finish the trailing ones, so a
// block costs its eight dependent steps, one block product and two CTA barriers. Returns 1 + the
// first column whose pivot was not positive, else 0 (the same in every thread). sc: kWarpScratch
// doubles.
// Omega update passes at N = 5003, l = 20 and N = 20000, l = 40: 12.9 and 22.1 us (15.7 and 28.0 with every
// warp factoring every block itself, unrolled a row a lane, and rounded
// reciprocals: their shuffles held one another up).
template <int NT>
__device__ __forceinline__ int chol_inverse(double* W, double* R, double* X, double* sc) {
  using T = Tall<NT>;
  constexpr int LD = T::LD;
  const int warp = threadIdx.x >> 5;
  double* Li = sc;                       // two 8 x 8: of the current and of the next block
  double* my = sc + 128 + warp * 64;     // kTallWarps x 8 x 8
  __shared__ int first_bad;
  for (int t = threadIdx.x; t < T::kSq; t += blockDim.x) R[t] = X[t] = 0.0;
  if (threadIdx.x == 0) first_bad = 0;
  __syncthreads();
  auto factor = [&](int b) {
    const int o = 8 * b * LD + 8 * b;
    const int bad = chol_block<LD>(W + o, R + o, X + o, Li + (b & 1) * 64);
    if (bad && threadIdx.x == 0 && first_bad == 0) first_bad = 8 * b + bad;
  };
#pragma unroll 1
  for (int b = -1; b + 1 < NT; ++b) {  // b = -1: the first diagonal block alone
    if (b >= 0 && b + 1 + warp < NT) {  // block row of R
      const int J = b + 1 + warp;
      double c[2] = {0.0, 0.0};
      block_mma<false>(c, Li + (b & 1) * 64, 8, W + 8 * b * LD + 8 * J, LD);
      block_store(c, R + 8 * b * LD + 8 * J, LD);
    }
    __syncthreads();
    // trailing tiles (I, J), b < I <= J, in rows: tile 0 is the next diagonal block, warp 0's
    const int rest = NT - 1 - b;
#pragma unroll 1
    for (int q = warp; b >= 0 && q < rest * rest; q += kTallWarps - 1) {
      const int I = b + 1 + q / rest, J = b + 1 + q % rest;
      if (J >= I) {
        double c[2];
        block_load(c, W + 8 * I * LD + 8 * J, LD);
        block_mma<true>(c, R + 8 * b * LD + 8 * I, LD, R + 8 * b * LD + 8 * J, LD, -1.0);
        block_store(c, W + 8 * I * LD + 8 * J, LD);
      }
      if (warp == 0) break;
    }
    if (warp == 0) {
      __syncwarp();
      factor(b + 1);
    }
    __syncthreads();
  }
  // block column J of the inverse by warp J: X_IJ = -X_II sum_{I < K <= J} R_IK X_KJ
  for (int J = warp; J < NT; J += kTallWarps)
#pragma unroll 1
    for (int I = J - 1; I >= 0; --I) {
      double c[2] = {0.0, 0.0}, g[2] = {0.0, 0.0};  // even and odd K apart: two chains of products
#pragma unroll 1
      for (int K = I + 1; K <= J; K += 2) {
        block_mma<false>(c, R + 8 * I * LD + 8 * K, LD, X + 8 * K * LD + 8 * J, LD);
        if (K < J) block_mma<false>(g, R + 8 * I * LD + 8 * (K + 1), LD, X + 8 * (K + 1) * LD + 8 * J, LD);
      }
      c[0] += g[0];
      c[1] += g[1];
      block_store(c, my, 8);
      __syncwarp();
      double e[2] = {0.0, 0.0};
      block_mma<false>(e, X + 8 * I * LD + 8 * I, LD, my, 8, -1.0);
      block_store(e, X + 8 * I * LD + 8 * J, LD);
      __syncwarp();
    }
  __syncthreads();
  return first_bad;
}

// C = A B for upper triangular A, B in shared memory (C may not alias them).
template <int NT>
__device__ __forceinline__ void upper_product(const double* A, const double* B, double* C) {
  constexpr int LD = Tall<NT>::LD;
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  for (int t = warp; t < NT * NT; t += kTallWarps) {
    const int I = t / NT, J = t - I * NT;
    double c[2] = {0.0, 0.0};
    for (int K = I; K <= J; ++K) block_mma<false>(c, A + 8 * I * LD + 8 * K, LD, B + 8 * K * LD + 8 * J, LD);
    block_store(c, C + 8 * I * LD + 8 * J, LD);
  }
  __syncthreads();
}

// Modified LU of the 8 x 8 block Tb (row stride LD): step j takes the pivot s = T[j][j],
// D_j = -sign(s) with sign(0) = +, and eliminates with the shifted pivot u = s - D_j (|u| >= 1).
// Writes D and the inverses of the two factors (Li unit lower, Ui upper, 8 x 8), which the
// elimination's row and column operations leave in two identities beside the block.
template <int LD>
__device__ __forceinline__ void signs_block(const double* Tb, double* D, double* Li, double* Ui) {
  const int lane = threadIdx.x & 31, r = lane & 7, g = lane >> 3, row0 = lane & 24;
  double t0 = Tb[r * LD + 2 * g], t1 = Tb[r * LD + 2 * g + 1], i0 = 1.0, i1 = 1.0;
  double y0 = r == 2 * g ? 1.0 : 0.0, y1 = r == 2 * g + 1 ? 1.0 : 0.0, z0 = y0, z1 = y1;
#pragma unroll 1
  for (int jj = 0; jj < 4; ++jj)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 2 * jj + h;
      const double tj = h ? t1 : t0, zj = h ? z1 : z0;
      const double piv = __shfl_sync(0xffffffffu, tj, 8 * jj + j);
      const double m = __shfl_sync(0xffffffffu, tj, 8 * jj + r), zr = __shfl_sync(0xffffffffu, zj, 8 * jj + r);
      const double w0 = __shfl_sync(0xffffffffu, t0, row0 + j), w1 = __shfl_sync(0xffffffffu, t1, row0 + j);
      const double v0 = __shfl_sync(0xffffffffu, y0, row0 + j), v1 = __shfl_sync(0xffffffffu, y1, row0 + j);
      const double di = piv >= 0.0 ? -1.0 : 1.0;
      if (lane == 0) D[j] = di;
      const double inv = fast_reciprocal(piv - di), f = r > j ? m * inv : 0.0;
      if (2 * g == j) i0 = inv;
      if (2 * g + 1 == j) i1 = inv;
      if (2 * g > j) {
        t0 -= f * w0;
        z0 -= zr * (w0 * inv);
      }
      if (2 * g + 1 > j) {
        t1 -= f * w1;
        z1 -= zr * (w1 * inv);
      }
      y0 -= f * v0;
      y1 -= f * v1;
    }
  Li[r * 8 + 2 * g] = y0;
  Li[r * 8 + 2 * g + 1] = y1;
  Ui[r * 8 + 2 * g] = z0 * i0;
  Ui[r * 8 + 2 * g + 1] = z1 * i1;
  __syncwarp();
}

// Householder column signs D (LT values, shared memory) of the thin QR whose orthonormal factor
// has the top l x l block T (shared memory, zero padded, overwritten): the modified LU of
// Ballard et al. 2015 in blocks of 8, warp 0 ahead of the others as in chol_inverse. sc:
// kWarpScratch doubles.
template <int NT>
__device__ __forceinline__ void householder_signs(double* T, double* D, double* sc) {
  constexpr int LD = Tall<NT>::LD;
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  auto factor = [&](int b) {
    signs_block<LD>(T + 8 * b * LD + 8 * b, D + 8 * b, sc + (b & 1) * 128, sc + (b & 1) * 128 + 64);
  };
#pragma unroll 1
  for (int b = -1; b + 1 < NT; ++b) {  // b = -1: the first diagonal block alone
    const double *Li = sc + (b & 1) * 128, *Ui = Li + 64;
    const int rest = NT - 1 - b;
#pragma unroll 1
    for (int q = warp; b >= 0 && q < 2 * rest; q += kTallWarps) {  // block row, then block column
      const bool row = q < rest;
      double* P = row ? T + 8 * b * LD + 8 * (b + 1 + q) : T + 8 * (b + 1 + q - rest) * LD + 8 * b;
      double c[2] = {0.0, 0.0};
      if (row)
        block_mma<false>(c, Li, 8, P, LD);
      else
        block_mma<false>(c, P, LD, Ui, 8);
      __syncwarp();
      block_store(c, P, LD);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = warp; b >= 0 && q < rest * rest; q += kTallWarps - 1) {  // tile 0 is warp 0's
      const int I = b + 1 + q / rest, J = b + 1 + q % rest;
      double c[2];
      block_load(c, T + 8 * I * LD + 8 * J, LD);
      block_mma<false>(c, T + 8 * I * LD + 8 * b, LD, T + 8 * b * LD + 8 * J, LD, -1.0);
      block_store(c, T + 8 * I * LD + 8 * J, LD);
      if (warp == 0) break;
    }
    if (warp == 0) {
      __syncwarp();
      factor(b + 1);
    }
    __syncthreads();
  }
}

// v[i] = sum_{b < n} x[b * stride + t + i * blockDim] in b order, t the thread, for the i with
// t + i * blockDim < count: the loads of four b of every element are issued before their adds.
template <int COUNT>
__device__ __forceinline__ void sum_parts(const double* x, int n, int64_t stride, double (&v)[(COUNT + kTallThreads - 1) / kTallThreads]) {
  constexpr int kPer = (COUNT + kTallThreads - 1) / kTallThreads;
#pragma unroll
  for (int i = 0; i < kPer; ++i) v[i] = 0.0;
  for (int b = 0; b < n; b += 4) {
    double w[4][kPer];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int e = threadIdx.x + i * kTallThreads;
        w[q][i] = b + q < n && e < COUNT ? x[(int64_t)(b + q) * stride + e] : 0.0;
      }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int i = 0; i < kPer; ++i) v[i] += w[q][i];
  }
}

// Cluster sum of the CTAs' part[n] (shared memory), in rank order, written to
// gout[cluster index * n + e]. Every CTA of the cluster calls it; the rank-r CTA sums the
// elements r * blockDim + t, ... through distributed shared memory. The second cluster barrier
// keeps each CTA's shared memory alive until the others have read it. The elements from nsum on
// are maxima (of non-negative values) instead of sums.
__device__ __forceinline__ void cluster_sum(const double* part, int n, int nsum, double* gout) {
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const int rank = (int)cl.block_rank();
  const int64_t cid = blockIdx.x / kTallCluster;
  for (int e = rank * blockDim.x + threadIdx.x; e < n; e += kTallCluster * blockDim.x) {
    double v[kTallCluster];
#pragma unroll
    for (int q = 0; q < kTallCluster; ++q) v[q] = cl.map_shared_rank(part, q)[e];
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kTallCluster; ++q) s = e < nsum ? s + v[q] : fmax(s, v[q]);
    gout[cid * n + e] = s;
  }
  cl.sync();
}

// Ticket: true in the CTA that finishes last (after a fence, so it sees every CTA's writes).
__device__ __forceinline__ bool last_cta(unsigned* counter) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(counter, 1u);
    last = (t == gridDim.x - 1);
    if (last) *counter = 0;  // ready for the next launch
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Clusters of kTallCluster CTAs of kernel (threads, smem bytes) that fit on the device at
// once, cached in the context by (kernel, key); 0 when the runtime cannot tell.
inline int resident_clusters(pcaone_ctx* c, const void* kernel, uint64_t key, int threads, size_t smem) {
  const auto k = std::make_pair(kernel, key);
  auto it = c->cluster_occupancy.find(k);
  if (it != c->cluster_occupancy.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kTallCluster * 64);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kTallCluster;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  c->cluster_occupancy[k] = n;
  return n;
}

}  // namespace pg

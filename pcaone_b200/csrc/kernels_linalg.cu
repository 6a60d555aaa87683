// FP64 kernels on tall row-major matrices (one sample or SNP per row, l <= kLmax columns) for the
// Omega update and the epoch tail: Gram products, products with a small factor, the l x l
// factorisations between them, column sums.
//
// CholeskyQR2 as a chain of passes (TallStep): every pass reads its rows once, applies the
// inverse factor of the pass before, sums the Gram matrix, and its last CTA factors and inverts
// it, so a pass is one launch. The passes over N x l matrices (0.2 - 6 MB, in L2) are bound by
// latency: launch, one round of loads, the reductions, and the l x l factorisation in one CTA.
// The passes over G (M x l) are bound by HBM.
#include "linalg.hpp"

#include <algorithm>

#include "pdl.hpp"
#include "tall.hpp"

namespace pg {

namespace {

template <int NT, bool RECT>
struct TallCfg {
  static constexpr int NB = (NT + 1) / 2;  // column tiles of B per pass over the rows
  static constexpr int kAcc = RECT ? NT * NB : Tall<NT>::kTiles;
  static constexpr int kRed = kTallWarps * kAcc * 64;
  static constexpr int kPost = RECT ? 0 : 4 * Tall<NT>::kSq + Tall<NT>::kWarpScratch;
  static constexpr size_t smem(bool prod) {
    return ((prod ? Tall<NT>::kSq : 0) + (size_t)kAcc * 64 + (kRed > kPost ? kRed : kPost)) * 8;
  }
};

// See TallStep. Warp w of a CTA takes the 8-row groups w, w + 8, ... of the CTA's rows; the
// next group's loads are in flight while the current one is multiplied (narrow matrices: the
// registers of wider ones go to the accumulators).
// Measured (ncu, us a launch; before: rows solved by substitution a thread each, 4 x 4 FMA tiles
// from shared memory, Cholesky with a barrier a column, separate factorisation launches):
//   Omega update without its operand copy, N = 20000, l = 40: 60 (was 176); N = 5003, l = 20: 36 (71)
//   whole update with the int8 operand: 72 (216) and 43 (98)
//   G passes of the epoch tail, M = 500000, l = 40: 66 + 99 (50 + 298, plus two Choleskys of 37);
//   the tail at M = 50000, N = 2000, l = 20: 71 an epoch (176)
template <int NT, bool PROD, bool RECT>
__global__ void __cluster_dims__(kTallCluster, 1, 1) __launch_bounds__(kTallThreads) k_tall(TallStep a) {
  using T = Tall<NT>;
  using C = TallCfg<NT, RECT>;
  constexpr int LD = T::LD, NB = C::NB, NACC = C::kAcc;
  static_assert(PROD || !RECT, "a cross pass reads the rows of a product");
  constexpr bool kPrefetch = NT <= 5;
  extern __shared__ __align__(16) double sm[];
  double* Rs = sm;
  double* cpart = sm + (PROD ? T::kSq : 0);
  double* red = cpart + NACC * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q4 = lane >> 2, r4 = lane & 3;
  const int l = a.l, lb = a.lb;
  pdl_begin();
  if constexpr (PROD) {
    load_square<NT>(a.Rinv, l, 0.0, Rs);
    __syncthreads();
  }
  int64_t r0, r1;
  tall_rows(a.n, blockIdx.x, gridDim.x, r0, r1);
  const int ncl = gridDim.x / kTallCluster;
  const int passes = RECT ? ((lb + 7) / 8 + NB - 1) / NB : 1;

  // this lane's 2 NT values of the rows base .. base + 7: the operand of the product (row q4,
  // columns 4 i + r4), or that of the Gram itself (rows r4 and r4 + 4, columns 8 t + q4)
  auto load = [&](int64_t base, double (&x)[2 * NT], bool sum) {
    auto row = [&](int i) { return base + (PROD ? q4 : 4 * (i & 1) + r4); };
    auto col = [&](int i) { return PROD ? 4 * i + r4 : 8 * (i >> 1) + q4; };
#pragma unroll
    for (int i = 0; i < 2 * NT; ++i) x[i] = row(i) < r1 && col(i) < l ? a.A[row(i) * l + col(i)] : 0.0;
    if constexpr (!PROD) {
      if (a.A2) {  // every load before the first store, which may alias for all the compiler knows
        double y[2 * NT];
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i) y[i] = row(i) < r1 && col(i) < l ? a.A2[row(i) * l + col(i)] : 0.0;
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i) {
          x[i] += y[i];
          if (sum && row(i) < r1 && col(i) < l) a.Asum[row(i) * l + col(i)] = x[i];
        }
      }
    }
  };

  for (int pass = 0; pass < passes; ++pass) {
    double acc[NACC][2];
#pragma unroll
    for (int t = 0; t < NACC; ++t) acc[t][0] = acc[t][1] = 0.0;
    double x[2 * NT], nx[kPrefetch ? 2 * NT : 1];
    int64_t base = r0 + 8 * warp;
    if (kPrefetch && base < r1) load(base, x, pass == 0);
    for (; base < r1; base += 8 * kTallWarps) {
      if constexpr (kPrefetch) {
        if (base + 8 * kTallWarps < r1) load(base + 8 * kTallWarps, nx, pass == 0);
      } else {
        load(base, x, pass == 0);
      }
      double f[NT][2];  // rows row(0), row(1) of column 8 t + q4
      if constexpr (PROD) {
#pragma unroll
        for (int t = 0; t < NT; ++t) f[t][0] = f[t][1] = 0.0;
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i)
#pragma unroll
          for (int t = i / 2; t < NT; ++t) dmma(f[t], Rs[(4 * i + r4) * LD + 8 * t + q4], x[i]);
        if (a.Q && pass == 0) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int64_t row = base + 2 * r4 + e;
#pragma unroll
            for (int t = 0; t < NT; ++t)
              if (row < r1 && 8 * t + q4 < l) a.Q[row * l + 8 * t + q4] = f[t][e];
          }
        }
      } else {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          f[t][0] = x[2 * t];
          f[t][1] = x[2 * t + 1];
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if constexpr (RECT) {
          const int64_t row = base + 2 * r4 + e;
          double b[NB];
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const int col = 8 * (pass * NB + j) + q4;
            b[j] = row < r1 && col < lb ? a.B[row * lb + col] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) dmma(acc[i * NB + j], f[i][e], b[j]);
        } else {
#pragma unroll
          for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = i; j < NT; ++j) dmma(acc[T::tile(i, j)], f[i][e], f[j][e]);
        }
      }
      if constexpr (kPrefetch) {
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i) x[i] = nx[i];
      }
    }
#pragma unroll
    for (int t = 0; t < NACC; ++t)
      *reinterpret_cast<double2*>(red + (warp * NACC + t) * 64 + q4 * 8 + 2 * r4) = make_double2(acc[t][0], acc[t][1]);
    __syncthreads();
    for (int e = threadIdx.x; e < NACC * 64; e += kTallThreads) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kTallWarps; ++w) s += red[w * NACC * 64 + e];
      cpart[e] = s;
    }
    cluster_sum(cpart, NACC * 64, NACC * 64, a.part + (int64_t)pass * ncl * NACC * 64);
  }
  if (!last_cta(a.counter)) return;

  constexpr int kPer = (NACC * 64 + kTallThreads - 1) / kTallThreads;
  if constexpr (RECT) {
    for (int pass = 0; pass < passes; ++pass) {
      double v[kPer];
      sum_parts<NACC * 64>(a.part + (int64_t)pass * ncl * NACC * 64, ncl, NACC * 64, v);
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int e = threadIdx.x + u * kTallThreads, t = e >> 6, i = t / NB, j = pass * NB + t % NB;
        const int row = 8 * i + ((e & 63) >> 3), col = 8 * j + (e & 7);
        if (e < NACC * 64 && row < l && col < lb) a.X[row * lb + col] = v[u];
      }
    }
  } else {
    double *W = red, *R = W + T::kSq, *X = R + T::kSq, *P = X + T::kSq, *sc = P + T::kSq;
    double v[kPer];
    sum_parts<NACC * 64>(a.part, ncl, NACC * 64, v);
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int e = threadIdx.x + u * kTallThreads;
      int i = 0, t = e >> 6;
      if (e >= NACC * 64) break;
      while (t >= NT - i) t -= NT - i++;
      const int row = 8 * i + ((e & 63) >> 3), col = 8 * (i + t) + (e & 7);
      W[row * LD + col] = (row < l && col < l) ? v[u] : (row == col ? 1.0 : 0.0);
    }
    if (a.Rprev) load_square<NT>(a.Rprev, l, 1.0, P);
    __syncthreads();
    const int bad = chol_inverse<NT>(W, R, X, sc);
    if (bad && threadIdx.x == 0) atomicMax(a.status, bad);
    if (a.R) store_square<NT>(R, l, a.R);
    if (a.Ri) store_square<NT>(X, l, a.Ri);
    if (a.Rprev) {
      upper_product<NT>(R, P, W);
      store_square<NT>(W, l, a.Racc);
      if (a.Rprev_inv) {
        __syncthreads();
        load_square<NT>(a.Rprev_inv, l, 1.0, P);
        upper_product<NT>(P, X, W);
        store_square<NT>(W, l, a.Racc_inv);
      }
    }
  }
}

template <int NT, bool PROD, bool RECT>
void launch_tall(pcaone_ctx* c, TallStep s) {
  constexpr size_t smem = TallCfg<NT, RECT>::smem(PROD);
  static_assert(smem <= 227 * 1024, "shared memory above the per-CTA limit");
  const void* kern = (const void*)k_tall<NT, PROD, RECT>;
  if (c->smem_attr_set.insert(kern).second)
    PG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // one 8-row group a warp (64 rows a CTA) while the clusters fit at once
  int cap = kTallMaxParts;
  const int resident = resident_clusters(c, kern, 0, kTallThreads, smem);
  if (resident > 0) cap = std::min(cap, resident);
  const int ncl = tall_clusters(s.n, cap);
  const int passes = RECT ? 2 : 1;
  s.part = tall_part(c, (size_t)passes * TallCfg<NT, RECT>::kAcc * 64);
  s.counter = tall_counter(c);
  launch_pdl(k_tall<NT, PROD, RECT>, ncl * kTallCluster, kTallThreads, smem, c->stream, s);
  c->launches++;
}

template <bool PROD, bool RECT>
void launch_tall_nt(pcaone_ctx* c, const TallStep& s) {
  switch ((s.l + 7) / 8) {
    case 1: launch_tall<1, PROD, RECT>(c, s); break;
    case 2: launch_tall<2, PROD, RECT>(c, s); break;
    case 3: launch_tall<3, PROD, RECT>(c, s); break;
    case 4: launch_tall<4, PROD, RECT>(c, s); break;
    case 5: launch_tall<5, PROD, RECT>(c, s); break;
    case 6: launch_tall<6, PROD, RECT>(c, s); break;
    case 7: launch_tall<7, PROD, RECT>(c, s); break;
    default: launch_tall<8, PROD, RECT>(c, s); break;
  }
}

// Forward substitution for one row: x R = a with R upper l x l staged by stage_r (row stride
// LMAX, so every R address is a constant offset; the diagonal slots hold 1 / R_jj, so the
// dependent chain has no division), x kept in registers (LMAX >= l; the loops unroll over LMAX
// and skip j >= l). Every element of a is read before out is written, so out may alias a.
template <int LMAX>
__device__ __forceinline__ void solve_row_upper(const double* a, const double* Rs, int l, double* out) {
  double x[LMAX];
#pragma unroll
  for (int j = 0; j < LMAX; ++j) {
    if (j < l) {
      double v = a[j];
#pragma unroll
      for (int k = 0; k < j; ++k) v -= x[k] * Rs[k * LMAX + j];
      x[j] = v * Rs[j * LMAX + j];
    } else {
      x[j] = 0.0;
    }
  }
#pragma unroll
  for (int j = 0; j < LMAX; ++j)
    if (j < l) out[j] = x[j];
}

// Copy R (l x l row-major, upper) into shared memory with row stride LMAX for
// solve_row_upper: the diagonal slots get 1 / R_jj.
template <int LMAX>
__device__ __forceinline__ void stage_r(const double* R, int l, double* Rs) {
  for (int t = threadIdx.x; t < l * l; t += blockDim.x) {
    const int i = t / l, j = t - i * l;
    Rs[i * LMAX + j] = i == j ? 1.0 / R[t] : R[t];
  }
}

// Q = A R^{-1} (row-wise forward substitution x R = a), R upper l x l. One thread per row;
// the row's unknowns stay in registers (LMAX >= l, loops unrolled over LMAX).
template <int LMAX>
__global__ void __launch_bounds__(128) k_trsm_right_upper(const double* A, const double* __restrict__ R, int l,
                                                          int64_t n, double* Q) {  // A may alias Q
  extern __shared__ double sr[];  // LMAX x LMAX
  stage_r<LMAX>(R, l, sr);
  __syncthreads();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  solve_row_upper<LMAX>(A + r * l, sr, l, Q + r * l);
}

// Column sums of A (n x l) into partials (grid.y = column).
__global__ void k_colsum_partial(const double* __restrict__ A, int l, int64_t n,
                                 double* __restrict__ part) {
  __shared__ double sm[256];
  const int col = blockIdx.y;
  double s = 0.0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x)
    s += A[r * l + col];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int st = blockDim.x / 2; st; st >>= 1) {
    if (threadIdx.x < st) sm[threadIdx.x] += sm[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(int64_t)col * gridDim.x + blockIdx.x] = sm[0];
}

__global__ void k_colsum_final(const double* __restrict__ part, int nblk, int l,
                               double* __restrict__ out) {
  int col = threadIdx.x;
  if (col >= l) return;
  double s = 0.0;
  for (int b = 0; b < nblk; ++b) s += part[(int64_t)col * nblk + b];
  out[col] = s;
}

// Y (n x kc) = X (n x l) * C (l x ldc, first kc columns), row-major; X row in registers.
template <int LMAX>
__global__ void __launch_bounds__(128) k_rowmat(const double* __restrict__ X, int l, const double* __restrict__ C,
                                                int ldc, int kc, int64_t n, double* __restrict__ Y) {
  extern __shared__ double sc[];
  for (int t = threadIdx.x; t < l * kc; t += blockDim.x) sc[t] = C[(t / kc) * ldc + t % kc];
  __syncthreads();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  const double* x = X + r * l;
  double xr[LMAX];
#pragma unroll
  for (int j = 0; j < LMAX; ++j) xr[j] = j < l ? x[j] : 0.0;
  for (int c = 0; c < kc; ++c) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < LMAX; ++j)
      if (j < l) s = fma(xr[j], sc[j * kc + c], s);
    Y[r * kc + c] = s;
  }
}

// 32 rows x all columns through shared memory, so that both sides are read and written in whole
// sectors (before, either the reads or the writes of a warp were l doubles apart).
constexpr int kLayoutRows = 32;
__global__ void __launch_bounds__(256) k_rowmajor(const double* __restrict__ cm, int64_t n, int l, int64_t npad,
                                                  const double* __restrict__ scale, double* __restrict__ out,
                                                  float* __restrict__ outf) {
  extern __shared__ double tile[];  // l x 33
  const int64_t i0 = (int64_t)blockIdx.x * kLayoutRows;
  const int rows = (int)(npad - i0 < kLayoutRows ? npad - i0 : kLayoutRows);
  for (int t = threadIdx.x; t < l * kLayoutRows; t += 256) {
    const int j = t >> 5, r = t & 31;
    const double v = i0 + r < n ? cm[j * n + i0 + r] : 0.0;
    tile[j * 33 + r] = scale ? v * scale[j] : v;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < rows * l; t += 256) {
    const int r = t / l, j = t - r * l;
    const double v = tile[j * 33 + r];
    out[i0 * l + t] = v;
    if (outf) outf[i0 * l + t] = (float)v;
  }
}

__global__ void __launch_bounds__(256) k_colmajor(const double* __restrict__ X, int64_t n, int l, int ld,
                                                  double* __restrict__ out) {
  extern __shared__ double tile[];  // l x 33
  const int64_t i0 = (int64_t)blockIdx.x * kLayoutRows;
  const int rows = (int)(n - i0 < kLayoutRows ? n - i0 : kLayoutRows);
  for (int t = threadIdx.x; t < rows * l; t += 256) {
    const int r = t / l, j = t - r * l;
    tile[j * 33 + r] = X[(i0 + r) * ld + j];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < l * kLayoutRows; t += 256) {
    const int j = t >> 5, r = t & 31;
    if (r < rows) out[j * n + i0 + r] = tile[j * 33 + r];
  }
}

}  // namespace

void to_rowmajor(pcaone_ctx* c, const double* cm, int64_t n, int l, int64_t npad, const double* scale, double* out,
                 float* outf) {
  const unsigned grid = (unsigned)((npad + kLayoutRows - 1) / kLayoutRows);
  if (!grid) return;
  k_rowmajor<<<grid, 256, (size_t)l * 33 * 8, c->stream>>>(cm, n, l, npad, scale, out, outf);
  PG_CHECK_LAUNCH();
  c->launches++;
}

void to_colmajor(pcaone_ctx* c, const double* X, int64_t n, int l, int ld, double* out) {
  const unsigned grid = (unsigned)((n + kLayoutRows - 1) / kLayoutRows);
  if (!grid) return;
  k_colmajor<<<grid, 256, (size_t)l * 33 * 8, c->stream>>>(X, n, l, ld, out);
  PG_CHECK_LAUNCH();
  c->launches++;
}

double* tall_part(pcaone_ctx* c, size_t doubles) {
  return (double*)scratch(c, "tall_part", (size_t)kTallMaxParts * doubles * 8);
}

void tall_step(pcaone_ctx* c, TallStep s) {
  PG_REQUIRE(s.l >= 1 && s.l <= kLmax && s.lb <= s.l, PCAONE_EBADARG, "sketch width out of range");
  PG_REQUIRE(s.n >= 1 && !(s.A2 && s.Rinv), PCAONE_EBADARG, "bad tall pass");
  PG_REQUIRE(!s.B || s.Q != s.A, PCAONE_EBADARG, "a cross pass may not overwrite its input");
  PG_REQUIRE(!s.B || s.Rinv, PCAONE_EBADARG, "a cross pass needs the inverse factor");
  if (s.B)
    launch_tall_nt<true, true>(c, s);
  else
    s.Rinv ? launch_tall_nt<true, false>(c, s) : launch_tall_nt<false, false>(c, s);
}

void trsm_right_upper(pcaone_ctx* c, const double* A, const double* R, int l, int64_t n, double* Q) {
  const dim3 grid((unsigned)((n + 127) / 128));
  if (l <= 16)
    k_trsm_right_upper<16><<<grid, 128, 16 * 16 * 8, c->stream>>>(A, R, l, n, Q);
  else if (l <= 32)
    k_trsm_right_upper<32><<<grid, 128, 32 * 32 * 8, c->stream>>>(A, R, l, n, Q);
  else if (l <= 48)
    k_trsm_right_upper<48><<<grid, 128, 48 * 48 * 8, c->stream>>>(A, R, l, n, Q);
  else
    k_trsm_right_upper<64><<<grid, 128, 64 * 64 * 8, c->stream>>>(A, R, l, n, Q);
  PG_CHECK_LAUNCH();
  c->launches++;
}

void colsum(pcaone_ctx* c, const double* A, int l, int64_t n, double* out) {
  const int nblk = 64;
  double* part = (double*)scratch(c, "colsum_part", (size_t)l * nblk * 8);
  k_colsum_partial<<<dim3(nblk, l), 256, 0, c->stream>>>(A, l, n, part);
  PG_CHECK_LAUNCH();
  k_colsum_final<<<1, 128, 0, c->stream>>>(part, nblk, l, out);
  PG_CHECK_LAUNCH();
  c->launches += 2;
}

void rowmat(pcaone_ctx* c, const double* X, int l, const double* C, int ldc, int kc, int64_t n, double* Y) {
  const dim3 grid((unsigned)((n + 127) / 128));
  const size_t smem = (size_t)l * kc * 8;
  if (l <= 16)
    k_rowmat<16><<<grid, 128, smem, c->stream>>>(X, l, C, ldc, kc, n, Y);
  else if (l <= 32)
    k_rowmat<32><<<grid, 128, smem, c->stream>>>(X, l, C, ldc, kc, n, Y);
  else if (l <= 48)
    k_rowmat<48><<<grid, 128, smem, c->stream>>>(X, l, C, ldc, kc, n, Y);
  else
    k_rowmat<64><<<grid, 128, smem, c->stream>>>(X, l, C, ldc, kc, n, Y);
  PG_CHECK_LAUNCH();
  c->launches++;
}

}  // namespace pg

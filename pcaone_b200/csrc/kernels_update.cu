// Fused Omega update: Omega = flipOmg(Omega_prev, thin Q of H) in four launches.
//
// Reference: the Householder QR + householderQ() + flipOmg block of the winSVD window loop
// (src/Halko.cpp:213-216) and of the Halko epochs (src/Halko.cpp:118-122, src/RSVD.hpp:81-90;
// the reference's Omega2 is a copy of the previous Omega).
//
//   tall_step  H = H1 + H2 (winSVD), Gram of H             last CTA: R1^-1
//   tall_step  Q1 = H R1^-1, Gram of Q1                    last CTA: R2^-1
//   k_flip     Q = Q1 R2^-1; per column sum |O - Q|, sum |O + Q|, sum Q, max |Q|; one extra
//              CTA: Householder signs D of Q                last CTA: multipliers m = +-D, column
//                                                           sums and maxima of Omega
//   k_apply    Omega = Q m and its operand copies (FP32, int8 pieces or split BF16)
//
// The maxima of k_flip are what the int8 pieces are scaled by, so k_apply writes them in the
// same pass (a separate maximum and quantisation pass over Omega before). The signs come from
// the modified LU of the top l x l block of Q (Ballard et al. 2015), which a CTA of its own
// works on while the others solve their rows.
#include <cuda_bf16.h>

#include <algorithm>

#include "linalg.hpp"
#include "pdl.hpp"
#include "quant.hpp"
#include "tall.hpp"
#include "tc_layout.hpp"
#include "update.hpp"

namespace pg {

namespace {

template <int NT>
struct FlipCfg {
  static constexpr int kRows = kTallWarps * 4 * Tall<NT>::LT;                           // warps' sums
  static constexpr int kSigns = Tall<NT>::kSq + Tall<NT>::LT + Tall<NT>::kWarpScratch;  // T, D, scratch
  static constexpr size_t smem = ((size_t)Tall<NT>::kSq + 4 * Tall<NT>::LT + (kRows > kSigns ? kRows : kSigns)) * 8;
};

// q = rows base .. base + 7 of Q1 R2^-1 (rows < r1): q[t][e] is row base + 2 r4 + e, column 8 t + q4.
template <int NT>
__device__ __forceinline__ void solve_rows(const double* Q1, const double* Rs, int64_t base, int64_t r1, int l,
                                           double (&q)[NT][2]) {
  const int lane = threadIdx.x & 31, q4 = lane >> 2, r4 = lane & 3;
  double x[2 * NT];
  const int64_t row = base + q4;
#pragma unroll
  for (int i = 0; i < 2 * NT; ++i) x[i] = row < r1 && 4 * i + r4 < l ? Q1[row * l + 4 * i + r4] : 0.0;
#pragma unroll
  for (int t = 0; t < NT; ++t) q[t][0] = q[t][1] = 0.0;
#pragma unroll
  for (int i = 0; i < 2 * NT; ++i)
#pragma unroll
    for (int t = i / 2; t < NT; ++t) dmma(q[t], Rs[(4 * i + r4) * Tall<NT>::LD + 8 * t + q4], x[i]);
}

// The flip sums are taken without the signs: A_c = sum |O - Q| and B_c = sum |O + Q| per
// column; with D_c = +1 they are |O - Q D| and |O + Q D|, with D_c = -1 swapped (the same values
// bit for bit). The sums and maxima of Q give those of Omega = +-Q. The last cluster holds the
// CTA that finds the signs and takes no rows. Q goes to a buffer of its own (the signs' CTA
// reads the rows of Q1 meanwhile).
template <int NT>
__global__ void __cluster_dims__(kTallCluster, 1, 1) __launch_bounds__(kTallThreads)
    k_flip(UpdateArgs a, const double* Q1, double* __restrict__ Q) {
  using T = Tall<NT>;
  constexpr int LT = T::LT, LD = T::LD;
  extern __shared__ __align__(16) double sm[];
  double* Rs = sm;
  double* cpart = Rs + T::kSq;  // LT each: A, B, sums, maxima
  double* red = cpart + 4 * LT;
  const int l = a.l, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q4 = lane >> 2, r4 = lane & 3;
  const int ctas = gridDim.x - kTallCluster;
  pdl_begin();
  load_square<NT>(a.R2i, l, 0.0, Rs);
  for (int t = threadIdx.x; t < 4 * LT; t += kTallThreads) cpart[t] = 0.0;
  __syncthreads();
  if ((int)blockIdx.x < ctas) {
    int64_t r0, r1;
    tall_rows(a.N, blockIdx.x, ctas, r0, r1);
    double sa[NT], sb[NT], sq[NT], mx[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) sa[t] = sb[t] = sq[t] = mx[t] = 0.0;
    for (int64_t base = r0 + 8 * warp; base < r1; base += 8 * kTallWarps) {
      double q[NT][2], o[NT][2];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int64_t row = base + 2 * r4 + e;
          o[t][e] = row < r1 && 8 * t + q4 < l ? a.Omg[row * l + 8 * t + q4] : 0.0;
        }
      solve_rows<NT>(Q1, Rs, base, r1, l, q);
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int64_t row = base + 2 * r4 + e;
          if (row < r1 && 8 * t + q4 < l) Q[row * l + 8 * t + q4] = q[t][e];
          sa[t] += fabs(o[t][e] - q[t][e]);
          sb[t] += fabs(o[t][e] + q[t][e]);
          sq[t] += q[t][e];
          mx[t] = fmax(mx[t], fabs(q[t][e]));
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
#pragma unroll
      for (int d = 1; d < 4; d <<= 1) {
        sa[t] += __shfl_xor_sync(0xffffffffu, sa[t], d);
        sb[t] += __shfl_xor_sync(0xffffffffu, sb[t], d);
        sq[t] += __shfl_xor_sync(0xffffffffu, sq[t], d);
        mx[t] = fmax(mx[t], __shfl_xor_sync(0xffffffffu, mx[t], d));
      }
      if (r4 == 0) {
        double* w = red + warp * 4 * LT + 8 * t + q4;
        w[0] = sa[t];
        w[LT] = sb[t];
        w[2 * LT] = sq[t];
        w[3 * LT] = mx[t];
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 4 * LT; e += kTallThreads) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kTallWarps; ++w) s = e < 3 * LT ? s + red[w * 4 * LT + e] : fmax(s, red[w * 4 * LT + e]);
      cpart[e] = s;
    }
  } else if ((int)blockIdx.x == ctas) {
    double *top = red, *D = top + T::kSq, *sc = D + LT;
    if (warp < NT) {  // the top l rows of Q, 8 a warp, zero past row l
      double q[NT][2];
      solve_rows<NT>(Q1, Rs, 8 * warp, l, l, q);
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int t = 0; t < NT; ++t) top[(8 * warp + 2 * r4 + e) * LD + 8 * t + q4] = q[t][e];
    }
    householder_signs<NT>(top, D, sc);
    for (int j = threadIdx.x; j < l; j += kTallThreads) a.D[j] = D[j];
  }
  cluster_sum(cpart, 4 * LT, 3 * LT, a.part);
  if (!last_cta(a.counter)) return;
  const int ncl = gridDim.x / kTallCluster;
  double* tot = red;  // the clusters' sums and maxima
  static_assert(4 * LT <= kTallThreads, "a thread per column statistic");
  if (threadIdx.x < 4 * LT) {
    double v = 0.0;
#pragma unroll 4
    for (int p = 0; p < ncl; ++p) {
      const double w = a.part[(int64_t)p * 4 * LT + threadIdx.x];
      v = (int)threadIdx.x < 3 * LT ? v + w : fmax(v, w);
    }
    tot[threadIdx.x] = v;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < l; j += kTallThreads) {
    const double A = tot[j], B = tot[LT + j], s = tot[2 * LT + j], top = tot[3 * LT + j];
    const double d = a.D[j];
    const double m = d > 0.0 ? A : B, p = d > 0.0 ? B : A;
    const double f = (m > 2.0 * p) ? -d : d;  // src/RSVD.hpp:85
    a.mult[j] = f;
    a.wsum[j] = f * s;
    if (a.i8.qmax) a.i8.qmax[j] = (unsigned long long)__double_as_longlong(top);
  }
}

// Omega = Q m over the 128 rows of a CTA (one K chunk of the int8 operand), coalesced.
constexpr int kApplyThreads = 512;
__global__ void __launch_bounds__(kApplyThreads) k_apply(UpdateArgs a, const double* Q) {
  extern __shared__ __align__(16) uint8_t img[];  // np x 128 bytes (int8 operand)
  __shared__ PieceTable tab;
  __shared__ double mult[kLmax];
  const int l = a.l, lp = i8_lp(l), np = i8_np(l);
  const int64_t base = (int64_t)blockIdx.x * kI8Chunk;
  const int rows = (int)(a.N - base < kI8Chunk ? (a.N > base ? a.N - base : 0) : kI8Chunk);
  pdl_begin();
  for (int j = threadIdx.x; j < l; j += kApplyThreads) mult[j] = a.mult[j];
  if (a.i8.bq) {
    tab.fill(a.i8.qmax, l, lp, a.i8.sig, blockIdx.x == 0);
    for (int t = threadIdx.x; t < np * 8; t += kApplyThreads)
      reinterpret_cast<uint4*>(img)[t] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  constexpr int kBatch = 4;  // loads before the stores, which may alias for all the compiler knows
  for (int t0 = threadIdx.x; t0 < rows * l; t0 += kBatch * kApplyThreads) {
    double q[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int t = t0 + u * kApplyThreads;
      q[u] = t < rows * l ? Q[base * l + t] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int t = t0 + u * kApplyThreads, rr = t / l, j = t - rr * l;
      if (t >= rows * l) break;
      const int64_t o = base * l + t;
      const double v = q[u] * mult[j];
      a.Omg[o] = v;
      if (a.Omgf) a.Omgf[o] = (float)v;
      if (a.i8.bq) tab.put(img, rr, j, lp, v);
      if (a.bt1) {
        const int64_t kp = tc_pos(base + rr);
        const float x = (float)v;
        const __nv_bfloat16 hi = __float2bfloat16_rn(x);
        a.bt1[bt_elem(j, kp, 2 * a.bt_half)] = hi;
        a.bt1[bt_elem(a.bt_half + j, kp, 2 * a.bt_half)] = __float2bfloat16_rn(x - __bfloat162float(hi));
      }
    }
  }
  if (!a.i8.bq) return;
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(a.i8.bq + (int64_t)blockIdx.x * np * 128);
  for (int t = threadIdx.x; t < np * 8; t += kApplyThreads) dst[t] = reinterpret_cast<const uint4*>(img)[t];
}

template <int NT>
void launch_flip(pcaone_ctx* c, UpdateArgs a, const double* Q1, double* Q) {
  constexpr size_t smem = FlipCfg<NT>::smem;
  static_assert(smem <= 227 * 1024, "shared memory above the per-CTA limit");
  const void* kern = (const void*)k_flip<NT>;
  if (c->smem_attr_set.insert(kern).second)
    PG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int cap = kTallMaxParts;
  const int resident = resident_clusters(c, kern, 0, kTallThreads, smem);
  if (resident > 0) cap = std::min(cap, resident);
  const int ncl = tall_clusters(a.N, cap - 1) + 1;  // one for the signs
  a.part = tall_part(c, 4 * Tall<NT>::LT);
  a.counter = tall_counter(c);
  launch_pdl(k_flip<NT>, ncl * kTallCluster, kTallThreads, smem, c->stream, a, Q1, Q);
  c->launches++;
}

}  // namespace

void fused_update(pcaone_ctx* c, UpdateArgs a) {
  PG_REQUIRE(a.l >= 1 && a.l <= kLmax, PCAONE_EBADARG, "sketch width out of range");
  TallStep s;
  s.n = a.N;
  s.l = a.l;
  s.status = a.status;
  s.A = a.H2 ? a.H1 : a.H;
  s.A2 = a.H2;
  s.Asum = a.H2 ? a.H : nullptr;
  s.Ri = a.R1i;
  tall_step(c, s);
  double* Q1 = (double*)scratch(c, "upd_Q1", (size_t)a.N * a.l * 8);
  TallStep t;
  t.n = a.N;
  t.l = a.l;
  t.status = a.status;
  t.A = a.H;
  t.Rinv = a.R1i;
  t.Q = Q1;
  t.Ri = a.R2i;
  tall_step(c, t);
  switch ((a.l + 7) / 8) {
    case 1: launch_flip<1>(c, a, Q1, a.Q); break;
    case 2: launch_flip<2>(c, a, Q1, a.Q); break;
    case 3: launch_flip<3>(c, a, Q1, a.Q); break;
    case 4: launch_flip<4>(c, a, Q1, a.Q); break;
    case 5: launch_flip<5>(c, a, Q1, a.Q); break;
    case 6: launch_flip<6>(c, a, Q1, a.Q); break;
    case 7: launch_flip<7>(c, a, Q1, a.Q); break;
    default: launch_flip<8>(c, a, Q1, a.Q); break;
  }
  const size_t img = a.i8.bq ? (size_t)i8_np(a.l) * 128 : 0;  // at most 24 KB
  launch_pdl(k_apply, (unsigned)(a.kpad / kI8Chunk), kApplyThreads, img, c->stream, a, a.Q);
  c->launches++;
}

}  // namespace pg

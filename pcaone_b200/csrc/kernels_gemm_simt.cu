// SIMT decode-GEMM (FP32 or FP64 FMA): the plain-precision GPU path.
//
//   out[s][r][c] = sum_{k in split s} val(code[r][k]) * B[k][c]
//
// with val(00, 01, 10, 11) = (2, 0, 1, 0): the A1 allele count, missing as 0. This is the
// raw product of the reference's G^T * Omega and G * G (src/Halko.cpp:123-124, 193-202);
// centring, scaling and the missing-entry terms are applied by the epilogue kernels.
//
// FP32 (k_decode_gemm): a CTA owns 128 rows; each thread owns 4 rows x 8 columns of the output; K
// is streamed in chunks of 64 codes (16 packed bytes per row) staged in shared memory together
// with the matching 64 rows of B.
// FP64 (k_decode_dmma, k_decode_dmv): the FP64 tensor tiles m8n8k4 for three columns or more,
// a matrix-vector form for one or two, where seven eighths of a tile would be padding.
//
// K may run over consecutive windows (KRun), so that a run of windows is one product: one launch
// with rows or K enough to fill the SMs instead of one per window (470 SNPs at M = 30011 in 64
// windows: four row tiles).
#include <algorithm>

#include "internal.hpp"
#include "pdl.hpp"
#include "rsvd.hpp"
#include "tall.hpp"

namespace pg {

namespace {

constexpr int kTR = 128;  // rows per CTA
constexpr int kKC = 64;   // codes per K chunk
constexpr int kRPT = 4;   // rows per thread
constexpr int kCW = 8;    // columns per thread

// Map 16 packed codes to their 2-bit values v = (1-b0)(2-b1): 00->2, 01->0, 10->1, 11->0.
__device__ __forceinline__ uint32_t map_values(uint32_t w) {
  uint32_t b0 = w & 0x55555555u, b1 = (w >> 1) & 0x55555555u;
  uint32_t v0 = b1 & ~b0;                 // het -> 1
  uint32_t v1 = ~(b0 | b1) & 0x55555555u; // hom A1 -> 2
  return v0 | (v1 << 1);
}

__device__ __forceinline__ float small_to_real(uint32_t x) { return __int_as_float(0x4B400000u | x) - 12582912.0f; }

// The K positions of a product: windows of cpw chunks of 64 codes (kpw = 64 cpw rows of B each),
// window w's codes win_bytes after those of window w - 1; position r of window w is valid when
// r < wlen and w * wlen + r < mtot (the others multiply nothing: B is not read there).
struct KRun {
  int64_t cpw, win_bytes, kpw, wlen, mtot;
  __device__ __forceinline__ int64_t valid(int64_t w) const { return min(wlen, mtot - w * wlen); }
};

// n bytes of asynchronous copy, zero-filled when !ok.
template <int kBytes>
__device__ __forceinline__ void cp_async_zfill(void* sdst, const void* gsrc, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(gsrc), "n"(kBytes), "r"(ok ? kBytes : 0)
               : "memory");
}

// The codes of a thread's four rows come straight from global memory (16 bytes a row and chunk)
// and B through two shared-memory buffers of 4-byte asynchronous copies, both one chunk ahead:
// with one to eight warps a CTA the copies' latency is what bounds it otherwise. FP32 sums run over
// kFlush chunks at most and then go to FP64 sums: over the 250000 SNPs of a long run in one
// go they would lose two digits (eigenvalues of 20000 x 500000: 1e-6 against 3e-8).
// Runs of a winSVD, M = 30011, N = 1502, l = 15, mean of 266 products: 12.8 us with splits
// down to one chunk (30.9 staged through registers with four chunks a split at least).
constexpr int kFlush = 4;
template <int G>
__global__ void __launch_bounds__(32 * G)
k_decode_gemm(const uint8_t* __restrict__ codes, uint32_t pitch, int64_t rows, int64_t chunks, KRun run,
              const float* B, int ldb, int l, int64_t kchunks_per_split,
              float* __restrict__ out) {
  constexpr int LDS = G * kCW;              // padded B columns in shared memory
  __shared__ __align__(16) float bsm[2][kKC * LDS];

  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * kTR + lane;
  const int64_t kc0 = (int64_t)blockIdx.y * kchunks_per_split, kc1 = min(kc0 + kchunks_per_split, chunks);
  const uint8_t* rowp[kRPT];
#pragma unroll
  for (int q = 0; q < kRPT; ++q) rowp[q] = codes + min(r0 + 32 * q, rows - 1) * (int64_t)pitch;
  for (int t = threadIdx.x; t < 2 * kKC * LDS; t += 32 * G) (&bsm[0][0])[t] = 0.f;  // padded columns stay zero
  pdl_begin();
  __syncthreads();
  auto issue = [&](int64_t kc, int buf) {
    const int64_t w = kc / run.cpw, k0 = (kc - w * run.cpw) * kKC, kv = run.valid(w) - k0;
    const float* Bc = B + (w * run.kpw + k0) * ldb;
    for (int t = threadIdx.x; t < kKC * l; t += 32 * G) {
      const int kk = t / l, cc = t - kk * l;
      const bool ok = kk < kv;
      cp_async_zfill<4>(&bsm[buf][kk * LDS + cc], ok ? Bc + (int64_t)kk * ldb + cc : B, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto fetch = [&](int64_t kc, uint4 (&x)[kRPT]) {
    const int64_t w = kc / run.cpw, o = w * run.win_bytes + (kc - w * run.cpw) * (kKC / 4);
#pragma unroll
    for (int q = 0; q < kRPT; ++q) x[q] = __ldg(reinterpret_cast<const uint4*>(rowp[q] + o));
  };

  float acc[kRPT][kCW];
  double sum[kRPT][kCW];
#pragma unroll
  for (int q = 0; q < kRPT; ++q)
#pragma unroll
    for (int c = 0; c < kCW; ++c) {
      acc[q][c] = 0.f;
      sum[q][c] = 0.0;
    }

  uint4 cur[kRPT], nxt[kRPT];
  if (kc0 < kc1) {
    issue(kc0, 0);
    fetch(kc0, cur);
  }
  for (int64_t kc = kc0; kc < kc1; ++kc) {
    const int buf = (int)(kc - kc0) & 1;
    if (kc + 1 < kc1) {
      issue(kc + 1, buf ^ 1);
      fetch(kc + 1, nxt);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const uint32_t* xw = reinterpret_cast<const uint32_t*>(cur);
#pragma unroll
    for (int wq = 0; wq < 4; ++wq) {
      uint32_t x[kRPT];
#pragma unroll
      for (int q = 0; q < kRPT; ++q) x[q] = map_values(xw[4 * q + wq]);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float4* brow = reinterpret_cast<const float4*>(&bsm[buf][(wq * 16 + e) * LDS + g * kCW]);
        const float4 b0 = brow[0], b1 = brow[1];
        const float b[kCW] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int q = 0; q < kRPT; ++q) {
          const float v = small_to_real((x[q] >> (2 * e)) & 3u);
#pragma unroll
          for (int c = 0; c < kCW; ++c) acc[q][c] = fmaf(v, b[c], acc[q][c]);
        }
      }
    }
    __syncthreads();  // the buffer is read before it is refilled
    if ((kc - kc0) % kFlush == kFlush - 1 || kc + 1 == kc1) {
#pragma unroll
      for (int q = 0; q < kRPT; ++q)
#pragma unroll
        for (int c = 0; c < kCW; ++c) {
          sum[q][c] += (double)acc[q][c];
          acc[q][c] = 0.f;
        }
    }
#pragma unroll
    for (int q = 0; q < kRPT; ++q) cur[q] = nxt[q];
  }
  float* o = out + (int64_t)blockIdx.y * rows * l;
#pragma unroll
  for (int q = 0; q < kRPT; ++q) {
    const int64_t r = r0 + 32 * q;
    if (r >= rows) continue;
#pragma unroll
    for (int c = 0; c < kCW; ++c) {
      const int col = g * kCW + c;
      if (col < l) o[r * l + col] = (float)sum[q][c];
    }
  }
}

// ---------------------------------------------------------------- FP64
// Value of raw code c (00 -> 2, 01 -> 0, 10 -> 1, 11 -> 0) as a double: its two high bytes are a
// byte lookup (2.0 = 0x4000.., 1.0 = 0x3FF0..), the rest is zero.
__device__ __forceinline__ double code_to_double(uint32_t c) {
  return __hiloint2double((int)__byte_perm(0x00004000u, 0x00003FF0u, c * 0x2200u + 0x1022u), 0);
}

// A CTA owns 128 rows, a warp 16 (two row tiles), NT column tiles of 8. A lane's A element of the
// four codes 4 s .. 4 s + 3 is code lane % 4 of byte s of row lane / 4, so the codes come
// straight from global memory (16 bytes a row and chunk, the next chunk's in flight) and a
// decoded value serves NT tensor tiles. B is staged 64 rows at a time in two buffers (8-byte
// asynchronous copies, row stride 4 mod 16 doubles: conflict-free 4 x 4 reads).
// Bound by the FP64 pipe for wide B. M = 60000, N = 5000, 10 columns: 459 us (689 as FMA tiles).
constexpr int kDmmaThreads = 256;
template <int NT>
__global__ void __launch_bounds__(kDmmaThreads)
k_decode_dmma(const uint8_t* __restrict__ codes, uint32_t pitch, int64_t rows, int64_t chunks, KRun run,
              const double* __restrict__ B, int ldb, int l, int64_t kchunks_per_split, double* __restrict__ out) {
  constexpr int LD = Tall<NT>::LD;
  extern __shared__ __align__(16) double bsm[];  // 2 x 64 x LD
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q4 = lane >> 2, r4 = lane & 3;
  const int64_t row0 = (int64_t)blockIdx.x * kTR + warp * 16 + q4;  // and row0 + 8
  const int64_t kc0 = (int64_t)blockIdx.y * kchunks_per_split, kc1 = min(kc0 + kchunks_per_split, chunks);
  const uint8_t* rowp[2] = {codes + min(row0, rows - 1) * (int64_t)pitch, codes + min(row0 + 8, rows - 1) * (int64_t)pitch};
  for (int t = threadIdx.x; t < 2 * kKC * LD; t += kDmmaThreads) bsm[t] = 0.0;  // padded columns stay zero
  __syncthreads();
  auto issue = [&](int64_t kc, int buf) {
    const int64_t w = kc / run.cpw, k0 = (kc - w * run.cpw) * kKC, kv = run.valid(w) - k0;
    const double* Bc = B + (w * run.kpw + k0) * ldb;
    double* dst = bsm + buf * kKC * LD;
    for (int t = threadIdx.x; t < kKC * l; t += kDmmaThreads) {
      const int kk = t / l, cc = t - kk * l;
      const bool ok = kk < kv;
      cp_async_zfill<8>(dst + kk * LD + cc, ok ? Bc + (int64_t)kk * ldb + cc : B, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto fetch = [&](int64_t kc, uint4 (&x)[2]) {
    const int64_t w = kc / run.cpw, o = w * run.win_bytes + (kc - w * run.cpw) * (kKC / 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) x[h] = __ldg(reinterpret_cast<const uint4*>(rowp[h] + o));
  };
  double acc[2][NT][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[h][t][0] = acc[h][t][1] = 0.0;
  uint4 cur[2], nxt[2];
  if (kc0 < kc1) {
    issue(kc0, 0);
    fetch(kc0, cur);
  }
  for (int64_t kc = kc0; kc < kc1; ++kc) {
    const int buf = (int)(kc - kc0) & 1;
    if (kc + 1 < kc1) {
      issue(kc + 1, buf ^ 1);
      fetch(kc + 1, nxt);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const double* bs = bsm + buf * kKC * LD + r4 * LD + q4;
    const uint32_t x[2][4] = {{cur[0].x >> (2 * r4), cur[0].y >> (2 * r4), cur[0].z >> (2 * r4), cur[0].w >> (2 * r4)},
                              {cur[1].x >> (2 * r4), cur[1].y >> (2 * r4), cur[1].z >> (2 * r4), cur[1].w >> (2 * r4)}};
#pragma unroll
    for (int s = 0; s < kKC / 4; ++s) {
      const double a0 = code_to_double((x[0][s >> 2] >> (8 * (s & 3))) & 3u);
      const double a1 = code_to_double((x[1][s >> 2] >> (8 * (s & 3))) & 3u);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const double b = bs[4 * s * LD + 8 * t];
        dmma(acc[0][t], a0, b);
        dmma(acc[1][t], a1, b);
      }
    }
    __syncthreads();  // the buffer is read before it is refilled
    cur[0] = nxt[0];
    cur[1] = nxt[1];
  }
  double* o = out + (int64_t)blockIdx.y * rows * l;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t row = row0 + 8 * h;
    if (row >= rows) continue;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = 8 * t + 2 * r4 + e;
        if (col < l) o[row * l + col] = acc[h][t][e];
      }
  }
}

// One or two columns: a warp owns kDmvRows rows, a lane 16 codes of each in a step of 512, and
// the matching values of B lie in shared memory in the lanes' order ([code of the word][word],
// 2048 rows of B at a time). A value of B read from shared memory serves kDmvRows rows (at one
// row a read, shared memory would hold the FP64 pipe to a quarter of its rate); the bound is
// the integer work of the decode. M = 60001, N = 3000, one column: 84 us (449 in the tiled form, 7 of 8 columns padding).
constexpr int kDmvThreads = 256, kDmvRows = 8, kDmvTile = kDmvThreads / 32 * kDmvRows, kDmvK = 2048;
template <int L>
__global__ void __launch_bounds__(kDmvThreads)
k_decode_dmv(const uint8_t* __restrict__ codes, uint32_t pitch, int64_t rows, int64_t chunks, KRun run,
             const double* __restrict__ B, int64_t kchunks_per_split, double* __restrict__ out) {
  constexpr int kSpan = kDmvK / kKC, kWords = kDmvK / 16 + 1;  // (+ 1: the transposing writes spread over the banks)
  __shared__ __align__(16) double bs[16 * kWords * L];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * kDmvTile + warp * kDmvRows;
  const int64_t kc0 = (int64_t)blockIdx.y * kchunks_per_split, kc1 = min(kc0 + kchunks_per_split, chunks);
  double acc[kDmvRows][L];
#pragma unroll
  for (int r = 0; r < kDmvRows; ++r)
#pragma unroll
    for (int c = 0; c < L; ++c) acc[r][c] = 0.0;
  for (int64_t kc = kc0; kc < kc1;) {
    // up to kSpan chunks that stay inside one window
    const int64_t w = kc / run.cpw, k0 = (kc - w * run.cpw) * kKC, kv = run.valid(w) - k0;
    const int64_t n = min((int64_t)kSpan, min(kc1 - kc, (w + 1) * run.cpw - kc));
    const int words = (int)n * (kKC / 16);
    const double* Bc = B + (w * run.kpw + k0) * L;
    __syncthreads();  // the previous values are used up
    for (int t = threadIdx.x; t < words * 16; t += kDmvThreads) {
      const int e = t & 15, wd = t >> 4;
#pragma unroll
      for (int c = 0; c < L; ++c) bs[(e * kWords + wd) * L + c] = t < kv ? Bc[t * L + c] : 0.0;
    }
    __syncthreads();
    const uint8_t* src = codes + w * run.win_bytes + (k0 >> 2);
    for (int wd = lane; wd < words; wd += 32) {
      uint32_t x[kDmvRows];
#pragma unroll
      for (int r = 0; r < kDmvRows; ++r)
        x[r] = __ldg(reinterpret_cast<const uint32_t*>(src + min(row0 + r, rows - 1) * (int64_t)pitch) + wd);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        double b[L];
#pragma unroll
        for (int c = 0; c < L; ++c) b[c] = bs[(e * kWords + wd) * L + c];
#pragma unroll
        for (int r = 0; r < kDmvRows; ++r) {
          const double v = code_to_double((x[r] >> (2 * e)) & 3u);
#pragma unroll
          for (int c = 0; c < L; ++c) acc[r][c] = fma(v, b[c], acc[r][c]);
        }
      }
    }
    kc += n;
  }
  double* o = out + (int64_t)blockIdx.y * rows * L;
#pragma unroll
  for (int r = 0; r < kDmvRows; ++r)
#pragma unroll
    for (int c = 0; c < L; ++c) {
      double v = acc[r][c];
      for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
      if (lane == 0 && row0 + r < rows) o[(row0 + r) * L + c] = v;
    }
}

KRun whole_k(int64_t K) {
  const int64_t chunks = (K + kKC - 1) / kKC;
  return KRun{chunks, 0, chunks * kKC, K, K};
}

void run_simt(pcaone_ctx* c, const uint8_t* codes, uint32_t pitch, int64_t rows, int64_t chunks, const KRun& run,
              const float* B, int ldb, int l, int ksplit, float* out) {
  const int64_t per = (chunks + ksplit - 1) / ksplit;
  const dim3 grid((unsigned)((rows + kTR - 1) / kTR), (unsigned)ksplit);
  auto go = [&](auto kern, int G) {
    launch_pdl(kern, grid, 32 * G, 0, c->stream, codes, pitch, rows, chunks, run, B, ldb, l, per, out);
  };
  switch ((l + kCW - 1) / kCW) {
    case 1: go(k_decode_gemm<1>, 1); break;
    case 2: go(k_decode_gemm<2>, 2); break;
    case 3: go(k_decode_gemm<3>, 3); break;
    case 4: go(k_decode_gemm<4>, 4); break;
    case 5: go(k_decode_gemm<5>, 5); break;
    case 6: go(k_decode_gemm<6>, 6); break;
    case 7: go(k_decode_gemm<7>, 7); break;
    default: go(k_decode_gemm<8>, 8); break;
  }
  PG_CHECK_LAUNCH();
  c->launches++;
  c->gemm_launches++;
}

void run_simt(pcaone_ctx* c, const uint8_t* codes, uint32_t pitch, int64_t rows, int64_t chunks, const KRun& run,
              const double* B, int ldb, int l, int ksplit, double* out) {
  PG_REQUIRE(ldb == l, PCAONE_EBADARG, "FP64 operand rows must be contiguous");
  const int64_t per = (chunks + ksplit - 1) / ksplit;
  if (l <= 2) {
    const dim3 grid((unsigned)((rows + kDmvTile - 1) / kDmvTile), (unsigned)ksplit);
    if (l == 1)
      k_decode_dmv<1><<<grid, kDmvThreads, 0, c->stream>>>(codes, pitch, rows, chunks, run, B, per, out);
    else
      k_decode_dmv<2><<<grid, kDmvThreads, 0, c->stream>>>(codes, pitch, rows, chunks, run, B, per, out);
  } else {
    const dim3 grid((unsigned)((rows + kTR - 1) / kTR), (unsigned)ksplit);
    auto go = [&](auto kern, int nt) {
      const size_t smem = (size_t)2 * kKC * (8 * nt + 4) * 8;
      if (c->smem_attr_set.insert((const void*)kern).second)
        PG_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      kern<<<grid, kDmmaThreads, smem, c->stream>>>(codes, pitch, rows, chunks, run, B, ldb, l, per, out);
    };
    switch ((l + 7) / 8) {
      case 1: go(k_decode_dmma<1>, 1); break;
      case 2: go(k_decode_dmma<2>, 2); break;
      case 3: go(k_decode_dmma<3>, 3); break;
      case 4: go(k_decode_dmma<4>, 4); break;
      case 5: go(k_decode_dmma<5>, 5); break;
      case 6: go(k_decode_dmma<6>, 6); break;
      case 7: go(k_decode_dmma<7>, 7); break;
      default: go(k_decode_dmma<8>, 8); break;
    }
  }
  PG_CHECK_LAUNCH();
  c->launches++;
  c->gemm_launches++;
}

}  // namespace

void launch_decode_gemm_simt(pcaone_ctx* c, const uint8_t* codes, uint32_t pitch, int64_t rows,
                             int64_t K, const float* B, int ldb, int l, int ksplit, float* out) {
  PG_REQUIRE(l >= 1 && l <= kLmax, PCAONE_EBADARG, "sketch width out of range");
  const KRun run = whole_k(K);
  run_simt(c, codes, pitch, rows, run.cpw, run, B, ldb, l, ksplit, out);
}

namespace {
template <typename T>
void simt_gemm(pcaone_ctx* c, const uint8_t* codes, uint32_t pitch, int64_t, int64_t rows, int64_t K,
               const T* B, int l, int ks, T* out) {
  PG_REQUIRE(l >= 1 && l <= kLmax, PCAONE_EBADARG, "sketch width out of range");
  const KRun run = whole_k(K);
  run_simt(c, codes, pitch, rows, run.cpw, run, B, l, l, ks, out);
}

// K splits: CTAs for about 16 warps an SM (FP32: 1 to 8 warps a CTA; FP64: 8). An FP32 warp's chunk
// is some 3500 instructions with no other warp to hide behind in a small product, so its
// splits go down to one chunk; the FP64 ones keep four, the matrix-vector form half a span of its
// staged B.
template <typename T>
int simt_ksplit(pcaone_ctx* c, int64_t rows, int64_t K, int l) {
  const bool dmv = sizeof(T) == 8 && l <= 2;
  const int64_t tile = dmv ? kDmvTile : kTR, warps = sizeof(T) == 8 ? 8 : (l + kCW - 1) / kCW;
  const int64_t tiles = (rows + tile - 1) / tile, chunks = (K + kKC - 1) / kKC;
  const int64_t ctas = std::max<int64_t>(2, (dmv ? 32 : 16) / warps);
  const int64_t want = (ctas * c->sm_count + tiles - 1) / tiles;
  const int64_t ks = std::max<int64_t>(1, std::min<int64_t>(want, chunks / (dmv ? kDmvK / kKC / 2 : sizeof(T) == 8 ? 4 : 1)));
  return (int)std::min<int64_t>(ks, 64);
}
void no_omega(pcaone_ctx*, const double*, int, int64_t) {}
template <typename T>
void no_b2(pcaone_ctx*, const T*, int, int64_t) {}

// ---- runs of consecutive windows [b0, b1): the first product's rows are the run's SNPs (contiguous
// records); the second product's K runs over the windows of the sample-major copies, each padded
// to its pitch.
int64_t simt_rows1(pcaone_ctx* c) { return (int64_t)c->win.blocksize; }
int64_t simt_k2(pcaone_ctx* c) { return (int64_t)c->win.pitch * 4; }
template <typename T>
int simt_ksplit_seg(pcaone_ctx* c, int which, int nw, int l) {
  return which == 1 ? simt_ksplit<T>(c, (int64_t)nw * (int64_t)c->win.blocksize, (int64_t)c->N, l)
                    : simt_ksplit<T>(c, (int64_t)c->N, (int64_t)nw * simt_k2(c), l);
}
template <typename T>
void simt_p1_seg(pcaone_ctx* c, int b0, int b1, const T* B, int l, int ks, T* out) {
  const int64_t s = (int64_t)c->win.start[b0], m = (int64_t)c->win.stop[b1 - 1] - s;
  simt_gemm<T>(c, c->streamed ? stream_codes(c, b0) : c->d_bed + s * (int64_t)c->pitch, c->pitch, s, m, (int64_t)c->N, B,
               l, ks, out);
}
template <typename T>
void simt_b2_seg(pcaone_ctx*, const T*, int, int, int) {}
template <typename T>
void simt_p2_seg(pcaone_ctx* c, int b0, int b1, const T* B2, int l, int ks, T* out) {
  const int64_t k2 = simt_k2(c), win_bytes = (int64_t)c->Npad * c->win.pitch;
  const KRun run{k2 / kKC, win_bytes, k2, (int64_t)c->win.blocksize, (int64_t)(c->win.stop[b1 - 1] - c->win.start[b0])};
  run_simt(c, c->streamed ? stream_codesT(c, b0) : c->d_bedT + b0 * win_bytes, c->win.pitch, (int64_t)c->N,
           (b1 - b0) * run.cpw, run, B2, l, l, ks, out);
}

template <typename T>
GemmFnT<T> simt_backend() {
  GemmFnT<T> f{simt_ksplit<T>, simt_gemm<T>, simt_gemm<T>, no_omega, no_b2<T>};
  f.seg_rows1 = simt_rows1;
  f.seg_k2 = simt_k2;
  f.seg_exact_rows = true;
  f.ksplit_seg = simt_ksplit_seg<T>;
  f.p1_seg = simt_p1_seg<T>;
  f.b2_seg = simt_b2_seg<T>;
  f.p2_seg = simt_p2_seg<T>;
  return f;
}
}  // namespace

GemmFnT<float> gemm_simt_float() { return simt_backend<float>(); }
GemmFnT<double> gemm_simt_double() { return simt_backend<double>(); }

}  // namespace pg

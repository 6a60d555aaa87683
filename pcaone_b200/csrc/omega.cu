// The reference's sketch Omega (RsvdOpData::initOmg, src/Halko.cpp:14-22): a
// std::default_random_engine (libstdc++ minstd_rand0) seeded with --seed, filled column-major
// with std::normal_distribution<double>(0, 1) draws (or uniform_real_distribution(-1, 1) with
// --rand 0). The result must be bit-identical to that sequential fill; it is generated here in
// parallel without changing a single draw:
//
//  * minstd_rand0 is x_{k+1} = 16807 x_k mod (2^31 - 1), so the state after d draws is
//    16807^d x_0 mod (2^31 - 1) (square-and-multiply), and an engine seeded with that state
//    continues the stream exactly;
//  * each uniform is std::generate_canonical<double, 53> of two draws, so a candidate pair of
//    the polar method (libstdc++ normal_distribution) consumes exactly four draws, and a
//    uniform_real_distribution value exactly two;
//  * the polar method keeps a candidate pair when 0 < x^2 + y^2 <= 1 and then returns y*m
//    followed by the saved x*m. So segments of candidate pairs are processed independently
//    (same expressions as libstdc++), and the accepted pairs are concatenated in segment
//    order, which is the sequential output order.
#include <algorithm>
#include <cmath>
#include <random>
#include <thread>
#include <vector>

#include "internal.hpp"
#include "rsvd.hpp"

namespace pg {

namespace {

constexpr uint64_t kM = 2147483647ull;  // minstd_rand0 modulus
constexpr uint64_t kA = 16807ull;       // minstd_rand0 multiplier

uint64_t pow_mod(uint64_t b, uint64_t e) {
  uint64_t r = 1;
  b %= kM;
  while (e) {
    if (e & 1) r = r * b % kM;
    b = b * b % kM;
    e >>= 1;
  }
  return r;
}

// Engine whose next draw is draw number d + 1 of the stream that starts at state x0.
std::minstd_rand0 engine_at(uint64_t x0, uint64_t d) {
  return std::minstd_rand0((std::minstd_rand0::result_type)(pow_mod(kA, d) * x0 % kM));
}

int worker_count() {
  const unsigned hc = std::thread::hardware_concurrency();
  return (int)std::max(1u, std::min(hc ? hc : 1u, 32u));
}

}  // namespace

void omega_host(int seed, int rand, uint64_t nrow, uint32_t ncol, double* out) {
  const uint64_t n = nrow * (uint64_t)ncol;
  if (n == 0) return;
  // libstdc++ linear_congruential_engine::seed: x0 = s mod m, or 1 when that is 0 (c = 0)
  const uint64_t s = (uint64_t)(std::minstd_rand0::result_type)seed;
  const uint64_t x0 = (s % kM) ? (s % kM) : 1;
  const int T = worker_count();
  if (!rand) {  // uniform_real_distribution(-1, 1): value i = canonical(draws 2i+1, 2i+2) * 2 - 1
    const uint64_t per = (n + T - 1) / T;
    std::vector<std::thread> th;
    for (int t = 0; t < T; ++t) {
      const uint64_t b = (uint64_t)t * per, e = std::min<uint64_t>(n, b + per);
      if (b >= e) break;
      th.emplace_back([=] {
        std::minstd_rand0 eng = engine_at(x0, 2 * b);
        std::uniform_real_distribution<double> d{-1, 1};
        for (uint64_t i = b; i < e; ++i) out[i] = d(eng);
      });
    }
    for (auto& x : th) x.join();
    return;
  }
  if (n < (1u << 16)) {  // small fills: the sequential distribution itself
    std::minstd_rand0 eng = engine_at(x0, 0);
    std::normal_distribution<double> d{0, 1};
    for (uint64_t i = 0; i < n; ++i) out[i] = d(eng);
    return;
  }
  // normal: one segment of candidate pairs per thread and round (4 draws per pair), sized so
  // that one round usually covers the n values (acceptance pi/4); further rounds continue
  // the stream where the last one stopped
  const uint64_t seg = ((uint64_t)((double)n / 2 / 0.75) / T) + 1024;
  std::vector<std::vector<double>> seg_out(T);
  uint64_t written = 0, next_pair = 0;
  while (written < n) {
    std::vector<std::thread> th;
    for (int t = 0; t < T; ++t) {
      const uint64_t p0 = next_pair + (uint64_t)t * seg;
      th.emplace_back([&, t, p0] {
        std::vector<double>& o = seg_out[t];
        o.clear();
        o.reserve(2 * seg);
        std::minstd_rand0 eng = engine_at(x0, p0 * 4);
        for (uint64_t p = 0; p < seg; ++p) {
          // the polar step of libstdc++ normal_distribution::operator(), same expressions
          const double x = 2.0 * std::generate_canonical<double, 53>(eng) - 1.0;
          const double y = 2.0 * std::generate_canonical<double, 53>(eng) - 1.0;
          const double r2 = x * x + y * y;
          if (r2 > 1.0 || r2 == 0.0) continue;
          const double mult = std::sqrt(-2 * std::log(r2) / r2);
          o.push_back(y * mult * 1.0 + 0.0);  // returned value, then the saved one
          o.push_back(x * mult * 1.0 + 0.0);
        }
      });
    }
    for (auto& x : th) x.join();
    for (int t = 0; t < T && written < n; ++t) {
      const uint64_t take = std::min<uint64_t>(n - written, seg_out[t].size());
      std::copy(seg_out[t].begin(), seg_out[t].begin() + take, out + written);
      written += take;
    }
    next_pair += (uint64_t)T * seg;
  }
}

// ---------------------------------------------------------------- on the device
// The same stream drawn by the GPU, a candidate pair (or a uniform value) a thread: the thread's
// engine state by square-and-multiply, the uniforms and the acceptance test in the same
// correctly rounded operations as above (no contraction), so exactly the same candidates are
// accepted; the accepted pairs are placed by an exclusive scan. sqrt is correctly rounded too;
// log is CUDA's (within one unit in the last place of the host library's). 20000 x 40 values took about
// 8 ms on the host's threads, their start and the upload included (winSVD 20000 x 500000 73.2 -> 65.3 ms
// without); fills below 65536 values,
// one thread of it, 25 ns a value.
namespace {

__device__ __forceinline__ uint32_t mod_m(uint64_t v) {  // v mod 2^31 - 1, v < 2^62
  v = (v & kM) + (v >> 31);
  v = (v & kM) + (v >> 31);
  return (uint32_t)(v >= kM ? v - kM : v);
}

// State after d draws from x0.
__device__ __forceinline__ uint32_t state_after(uint32_t x0, uint64_t d) {
  uint32_t r = x0, b = (uint32_t)kA;
  for (; d; d >>= 1) {
    if (d & 1) r = mod_m((uint64_t)r * b);
    b = mod_m((uint64_t)b * b);
  }
  return r;
}

// std::generate_canonical<double, 53> of the next two draws.
__device__ __forceinline__ double canonical(uint32_t& x) {
  constexpr double kR = 2147483646.0;  // engine range
  x = mod_m((uint64_t)x * kA);
  const double lo = (double)(x - 1);
  x = mod_m((uint64_t)x * kA);
  const double u = __ddiv_rn(__dadd_rn(lo, __dmul_rn((double)(x - 1), kR)), __dmul_rn(kR, kR));
  return u < 1.0 ? u : 1.0 - 0x1p-53;
}

__device__ __forceinline__ double symmetric(uint32_t& x) { return __dadd_rn(__dmul_rn(2.0, canonical(x)), -1.0); }

// Value i of the column-major fill -> row-major Omega (and its FP32 copy).
__device__ __forceinline__ void put_value(uint64_t i, uint64_t n, uint64_t nrow, int l, double v, double* O, float* Of) {
  if (i >= n) return;
  const uint64_t c = i / nrow, r = i - c * nrow;
  O[r * l + c] = v;
  if (Of) Of[r * l + c] = (float)v;
}

constexpr int kPairsPerCta = 256;
// base null: the accepted pairs of each CTA; else the pairs' values from base[CTA] on.
__global__ void __launch_bounds__(kPairsPerCta) k_omega_normal(uint32_t x0, uint64_t n, uint64_t nrow, int l,
                                                               const int64_t* __restrict__ base,
                                                               int64_t* __restrict__ count, double* __restrict__ O,
                                                               float* __restrict__ Of) {
  __shared__ int warp_sum[kPairsPerCta / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t s = state_after(x0, 4 * ((uint64_t)blockIdx.x * kPairsPerCta + threadIdx.x));
  const double x = symmetric(s), y = symmetric(s);
  const double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
  const bool ok = !(r2 > 1.0 || r2 == 0.0);
  const unsigned m = __ballot_sync(0xffffffffu, ok);
  if (lane == 0) warp_sum[warp] = __popc(m);
  __syncthreads();
  int before = __popc(m & ((1u << lane) - 1)), total = 0;
  for (int w = 0; w < kPairsPerCta / 32; ++w) {
    if (w < warp) before += warp_sum[w];
    total += warp_sum[w];
  }
  if (!base) {
    if (threadIdx.x == 0) count[blockIdx.x] = total;
    return;
  }
  if (!ok) return;
  const double mult = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, log(r2)), r2));
  const uint64_t i = 2 * (uint64_t)(base[blockIdx.x] + before);
  put_value(i, n, nrow, l, __dmul_rn(y, mult), O, Of);
  put_value(i + 1, n, nrow, l, __dmul_rn(x, mult), O, Of);
}

__global__ void __launch_bounds__(256) k_omega_uniform(uint32_t x0, uint64_t n, uint64_t nrow, int l,
                                                       double* __restrict__ O, float* __restrict__ Of) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  uint32_t s = state_after(x0, 2 * i);
  put_value(i, n, nrow, l, symmetric(s), O, Of);
}

}  // namespace

void omega_device(pcaone_ctx* c, int seed, int rand, uint64_t nrow, int l, uint64_t npad, double* O, float* Of) {
  const uint64_t n = nrow * (uint64_t)l;
  const uint64_t s = (uint64_t)(std::minstd_rand0::result_type)seed;
  const uint32_t x0 = (uint32_t)((s % kM) ? (s % kM) : 1);
  const size_t pad = (size_t)(npad - nrow) * l;
  PG_CUDA(cudaMemsetAsync(O + n, 0, pad * 8, c->stream));
  if (Of) PG_CUDA(cudaMemsetAsync(Of + n, 0, pad * 4, c->stream));
  if (!rand) {
    k_omega_uniform<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(x0, n, nrow, l, O, Of);
    PG_CHECK_LAUNCH();
    c->launches++;
    return;
  }
  // candidates for n / 2 accepted pairs at acceptance pi / 4 with more than 3% to spare, and again
  // twice as many in the case that was not enough
  for (uint64_t pairs = (uint64_t)((double)n / 2 / 0.76) + 1024;; pairs *= 2) {
    const unsigned ctas = (unsigned)((pairs + kPairsPerCta - 1) / kPairsPerCta);
    int64_t* cnt = (int64_t*)scratch(c, "omega_count", (size_t)ctas * 8);
    int64_t* base = (int64_t*)scratch(c, "omega_base", ((size_t)ctas + 1) * 8);
    k_omega_normal<<<ctas, kPairsPerCta, 0, c->stream>>>(x0, n, nrow, l, nullptr, cnt, O, Of);
    PG_CHECK_LAUNCH();
    c->launches++;
    if ((uint64_t)scan_counts(c, cnt, ctas, base) * 2 < n) continue;
    k_omega_normal<<<ctas, kPairsPerCta, 0, c->stream>>>(x0, n, nrow, l, base, cnt, O, Of);
    PG_CHECK_LAUNCH();
    c->launches++;
    return;
  }
}

}  // namespace pg

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
#include "linalg.hpp"
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
// The same fill, bit for bit, with all but the logarithms done by the GPU, a candidate pair (or a
// uniform value) a thread: the thread's engine state by square-and-multiply, the uniforms and the
// acceptance test in the same correctly rounded operations as above (no contraction), so
// exactly the same candidates are accepted; the accepted pairs are placed by an exclusive scan.
// The logarithm of the polar step is the host library's, which is neither correctly rounded nor the
// GPU's: the GPU takes it in two doubles, far beyond the last place, and rounds it where the
// host's cannot differ (rounds_surely); the other pairs, one in seventeen, go to the host for their
// factors. RSVD of two epochs, 20000 x 2000, l = 40: 2.3 ms (1.95 with the GPU's own log, 6.4 with the
// whole fill on the host's threads); 2000 x 50000, l = 20: 1.09 (1.04, 1.86). Fills up to 4096 values
// take 25 ns a value on one host thread.
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

// Position of value i of the column-major fill in row-major Omega.
__device__ __forceinline__ uint64_t place(uint64_t i, uint64_t nrow, int l) {
  const uint64_t c = i / nrow;
  return (i - c * nrow) * l + c;
}

// Fills up to this size are quicker on one host thread than two passes, a scan and a round trip.
constexpr uint64_t kHostFill = 4096;
constexpr int kPairsPerCta = 256;
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {  // Knuth
  s = __dadd_rn(a, b);
  const double t = __dadd_rn(s, -a);
  e = __dadd_rn(__dadd_rn(a, -__dadd_rn(s, -t)), __dadd_rn(b, -t));
}
__device__ __forceinline__ void two_prod(double a, double b, double& p, double& e) {
  p = __dmul_rn(a, b);
  e = fma(a, b, -p);
}

// log(x) = hi + lo for x in (0, 1], hi the nearest double: x = 2^k m with m in (sqrt(1/2), sqrt(2)],
// log m = 2 atanh(s), s = (m - 1) / (m + 1), by the series s + s^3 / 3 + s^5 / 5 + ... with its
// first two terms in two doubles. Error below 0.0012 units in the last place of hi (against 113-bit
// logarithms of 2.7 million values, to 2^-130 and next to 1).
__device__ __forceinline__ void log_parts(double x, double& hi, double& lo) {
  const long long bits = __double_as_longlong(x);
  int k = (int)(bits >> 52) - 1023;
  double m = __longlong_as_double((bits & 0xfffffffffffffll) | 0x3ff0000000000000ll);
  if (m > 1.4142135623730951) {
    m *= 0.5;
    ++k;
  }
  double den, den_lo, z, z_lo, a, a_lo, t, t_lo, p, p_lo, h, h_lo, c, c_lo, r, r_lo;
  two_sum(m, 1.0, den, den_lo);
  const double num = m - 1.0;  // exact
  const double s = __ddiv_rn(num, den), s_lo = __ddiv_rn(fma(-s, den_lo, fma(-s, den, num)), den);
  two_prod(s, s, z, z_lo);
  z_lo = fma(2.0 * s, s_lo, z_lo);
  double q = 0.0;  // 1/5 + z/7 + ... + z^12/29
#pragma unroll
  for (int j = 14; j >= 2; --j) q = fma(q, z, 1.0 / (2 * j + 1));
  two_prod(z, 0x1.5555555555555p-2, a, a_lo);  // z / 3
  a_lo = fma(z, 0x1.5555555555555p-56, fma(z_lo, 0x1.5555555555555p-2, a_lo));
  two_sum(a, __dmul_rn(__dmul_rn(z, z), q), t, t_lo);
  t_lo = __dadd_rn(t_lo, a_lo);
  two_prod(s, t, p, p_lo);
  p_lo = fma(s, t_lo, fma(s_lo, t, p_lo));
  two_sum(s, p, h, h_lo);
  h_lo = __dadd_rn(h_lo, __dadd_rn(p_lo, s_lo));
  two_prod((double)k, 0x1.62e42fefa39efp-1, c, c_lo);  // k log 2
  c_lo = fma((double)k, 0x1.abc9e3b39803fp-56, c_lo);
  two_sum(c, 2.0 * h, r, r_lo);
  two_sum(r, __dadd_rn(r_lo, fma(2.0, h_lo, c_lo)), hi, lo);
}

// Whether a library whose logarithms are within 0.53 units in the last place of the true ones (glibc:
// below 0.52) can return nothing but hi (hi not a power of two: the units below are half as large).
constexpr double kSure = 0.47;
__device__ __forceinline__ bool rounds_surely(double hi, double lo) {
  const long long bits = __double_as_longlong(hi);
  if (hi == 0.0) return lo == 0.0;
  const double unit = __longlong_as_double((bits & 0x7ff0000000000000ll) - (52ll << 52));
  return fabs(lo) <= kSure * unit && (bits & 0xfffffffffffffll) != 0;
}

__device__ __forceinline__ void put(uint64_t i, uint64_t nrow, int l, double v, double* O, float* Of) {
  const uint64_t at = place(i, nrow, l);
  O[at] = v;
  if (Of) Of[at] = (float)v;
}
// A value times its pair's factor (+ 0.0 as in the host's expression: no negative zeros).
__device__ __forceinline__ double scaled(double v, double factor) { return __dadd_rn(__dmul_rn(v, factor), 0.0); }

// Pairs left to the host, a list headed by their number: index and r^2, in its place later the factor.
struct OpenPair {
  uint64_t pair;
  double rr;
};

// base null: the accepted pairs of each CTA; else their values from pair base[CTA] on, or, for the open
// pairs, the values before the factor and an entry of the list.
__global__ void __launch_bounds__(kPairsPerCta) k_omega_pairs(uint32_t x0, uint64_t n, uint64_t nrow, int l,
                                                              const int64_t* __restrict__ base,
                                                              int64_t* __restrict__ count, double* __restrict__ O,
                                                              float* __restrict__ Of, OpenPair* open) {
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
  const uint64_t pair = (uint64_t)(base[blockIdx.x] + before);
  if (!ok || 2 * pair >= n) return;
  double hi, lo, factor = 1.0;
  log_parts(r2, hi, lo);
  if (rounds_surely(hi, lo))
    factor = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, hi), r2));
  else
    open[1 + atomicAdd((unsigned long long*)&open->pair, 1ull)] = OpenPair{pair, r2};
  put(2 * pair, nrow, l, scaled(y, factor), O, Of);
  if (2 * pair + 1 < n) put(2 * pair + 1, nrow, l, scaled(x, factor), O, Of);
}

// The values of the open pairs times the host's factors.
__global__ void __launch_bounds__(256) k_omega_open(uint64_t m, uint64_t n, uint64_t nrow, int l,
                                                    const OpenPair* __restrict__ open, double* __restrict__ O,
                                                    float* __restrict__ Of) {
  const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (t >= m) return;
  const OpenPair e = open[1 + t];
  put(2 * e.pair, nrow, l, scaled(O[place(2 * e.pair, nrow, l)], e.rr), O, Of);
  if (2 * e.pair + 1 < n) put(2 * e.pair + 1, nrow, l, scaled(O[place(2 * e.pair + 1, nrow, l)], e.rr), O, Of);
}

__global__ void __launch_bounds__(256) k_omega_uniform(uint32_t x0, uint64_t n, uint64_t nrow, int l,
                                                       double* __restrict__ O, float* __restrict__ Of) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  uint32_t s = state_after(x0, 2 * i);
  put(i, nrow, l, symmetric(s), O, Of);
}

}  // namespace

void omega_device(pcaone_ctx* c, int seed, int rand, uint64_t nrow, int l, uint64_t npad, double* O, float* Of) {
  const uint64_t n = nrow * (uint64_t)l;
  if (rand && n <= kHostFill) {
    std::vector<double> host(n);
    omega_host(seed, rand, nrow, (uint32_t)l, host.data());
    double* cm = (double*)scratch(c, "r_omg_cm", n * 8);
    PG_CUDA(cudaMemcpyAsync(cm, host.data(), n * 8, cudaMemcpyHostToDevice, c->stream));
    to_rowmajor(c, cm, (int64_t)nrow, l, (int64_t)npad, nullptr, O, Of);
    return;  // a copy of pageable memory has left it when it returns
  }
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
  const uint64_t kept = (n + 1) / 2;
  OpenPair* open = nullptr;
  for (uint64_t pairs = (uint64_t)((double)n / 2 / 0.76) + 1024;; pairs *= 2) {
    const unsigned ctas = (unsigned)((pairs + kPairsPerCta - 1) / kPairsPerCta);
    // one buffer for the list and the counts: each allocation is felt in a context's first call
    const size_t list = round_up((1 + kept) * sizeof(OpenPair), 256), counts = round_up((size_t)ctas * 8, 256);
    char* work = (char*)scratch(c, "omega_work", list + counts + ((size_t)ctas + 1) * 8);
    open = (OpenPair*)work;
    int64_t *cnt = (int64_t*)(work + list), *base = (int64_t*)(work + list + counts);
    k_omega_pairs<<<ctas, kPairsPerCta, 0, c->stream>>>(x0, n, nrow, l, nullptr, cnt, O, Of, open);
    PG_CHECK_LAUNCH();
    c->launches++;
    if ((uint64_t)scan_counts(c, cnt, ctas, base) < kept) continue;
    PG_CUDA(cudaMemsetAsync(open, 0, sizeof(OpenPair), c->stream));
    k_omega_pairs<<<ctas, kPairsPerCta, 0, c->stream>>>(x0, n, nrow, l, base, cnt, O, Of, open);
    PG_CHECK_LAUNCH();
    c->launches++;
    break;
  }
  // the list in one copy (of twice the expected length), its rest in another where that was short
  std::vector<OpenPair> host(1 + std::min(kept, kept / 8 + 64));
  PG_CUDA(cudaMemcpyAsync(host.data(), open, host.size() * sizeof(OpenPair), cudaMemcpyDeviceToHost, c->stream));
  PG_CUDA(cudaStreamSynchronize(c->stream));
  const uint64_t m = host[0].pair, have = std::min<uint64_t>(m, host.size() - 1);
  if (m == 0) return;
  host.resize(1 + m);
  if (m > have) {
    PG_CUDA(cudaMemcpyAsync(&host[1 + have], open + 1 + have, (m - have) * sizeof(OpenPair), cudaMemcpyDeviceToHost,
                            c->stream));
    PG_CUDA(cudaStreamSynchronize(c->stream));
  }
  for (uint64_t t = 1; t <= m; ++t) host[t].rr = std::sqrt(-2 * std::log(host[t].rr) / host[t].rr);
  PG_CUDA(cudaMemcpyAsync(open + 1, &host[1], m * sizeof(OpenPair), cudaMemcpyHostToDevice, c->stream));
  k_omega_open<<<(unsigned)((m + 255) / 256), 256, 0, c->stream>>>(m, n, nrow, l, open, O, Of);
  PG_CHECK_LAUNCH();
  c->launches++;
}

}  // namespace pg

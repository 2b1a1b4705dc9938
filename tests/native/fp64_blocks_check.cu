// Check of the FP64 lane's building blocks (rg_fp64.cuh) on the device: each returns the bits of what it
// stands in for.  Quotients are tried on random arguments over the ranges that the lane divides in and on
// the hardest ones a divisor has, whose exact quotient lies within a unit of the remainder from a midpoint
// of two doubles: n·2^53 - (2k + 1)·d = r for |r| = 1, 3 or 5 in the integers of the significands, which
// the divisor's inverse modulo 2^53 gives.  Inverse normals are tried on every 32-bit point.  Built with
// -fmad=false like the lane and run by tests/test_fp64_blocks_gpu.py.
#include <cstdio>
#include "rg_fp64.cuh"
using namespace rg;

enum { kRandom, kHard, kHardTop, kKnown, kExp, kLog, kExact, kCentral, kTail, kChecks };

struct Bad {
  unsigned long long count[kChecks];
  double a[kChecks], b[kChecks];
};

__device__ uint64_t mix(uint64_t x) {  // SplitMix64's output function
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}
__device__ double uniform(uint64_t key, double lo, double hi) { return lo + (hi - lo) * ((double)(mix(key) >> 11) * 0x1p-53); }
__device__ void check(Bad* bad, int what, double got, double want, double a, double b) {
  if (__double_as_longlong(got) == __double_as_longlong(want)) return;
  if (atomicAdd(&bad->count[what], 1ULL) == 0) {
    bad->a[what] = a;
    bad->b[what] = b;
  }
}

// The quotients of divisor d (in [1, 2)) that are hardest to round.
__device__ void hard_quotients(Bad* bad, int what, double d) {
  const uint64_t D = ((uint64_t)__double_as_longlong(d) & 0xfffffffffffffULL) | 0x10000000000000ULL;
  if (!(D & 1)) return;  // an even divisor's quotients keep farther from the midpoints
  const uint64_t mask = (1ULL << 53) - 1;
  uint64_t inv = D;  // Newton modulo a power of two: 3 bits of the inverse, doubled five times
  for (int i = 0; i < 5; ++i) inv *= 2 - D * inv;
  for (int r = -5; r <= 5; r += 2) {
    const uint64_t odd = (((uint64_t)(int64_t)-r * inv) & mask) + (1ULL << 53);  // 2k + 1
    // n = (odd·D + r) / 2^53 in 128 bits
    const uint64_t lo = odd * D, hi = __umul64hi(odd, D);
    const uint64_t lo2 = lo + (uint64_t)(int64_t)r, hi2 = hi + (r < 0 ? (lo2 > lo ? -1ULL : 0ULL) : (lo2 < lo ? 1ULL : 0ULL));
    if (lo2 & mask) continue;
    const uint64_t n = (hi2 << 11) | (lo2 >> 53);
    if (n >> 53 && (n & 1)) continue;  // not a double
    const double x = (double)n * 0x1p-52;
    check(bad, what, divide(x, d), x / d, x, d);
    check(bad, what, divide(-x * 0x1p-30, 0.5 * d), (-x * 0x1p-30) / (0.5 * d), x, d);
    check(bad, kKnown, divide_by(x, d, 1.0 / d), x / d, x, d);
  }
}

__global__ void quotients(Bad* bad, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    // the logarithm's f / (2 + f), Acklam's ratio, an axis cell
    const double f = uniform(4 * i, -0.2929, 0.4143), d = 2.0 + f;
    check(bad, kRandom, divide(f, d), f / d, f, d);
    const double num = uniform(4 * i + 1, -2.6, 2.6), den = uniform(4 * i + 2, 0.05, 1.0);
    check(bad, kRandom, divide(num, den), num / den, num, den);
    const double cell = uniform(4 * i + 3, 1e-4, 0.5), x = cell * uniform(4 * i + 1, 0.0, 1.0);
    check(bad, kRandom, divide_by(x, cell, 1.0 / cell), x / cell, x, cell);
    hard_quotients(bad, kHard, uniform(4 * i + 2, 1.0, 2.0));
    // divisors next below two, whose reciprocals lie next to midpoints, and within 2^-13 of it
    hard_quotients(bad, kHardTop, 2.0 - (double)(2 * (i & 0x3fffffULL) + 1) * 0x1p-52);
    hard_quotients(bad, kHardTop, 2.0 - uniform(4 * i, 0.0, 0x1p-11));
  }
}

__global__ void functions(Bad* bad, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const double wide = (i & 1) ? 800.0 : 0.5, x = uniform(3 * i, -wide, wide);
    check(bad, kExp, fast_exp64(x), rg_exp64(x), x, 0.0);
    // positive normals of every exponent, near one and near its reduction's edges
    const uint64_t h = mix(3 * i + 1);
    double y = __longlong_as_double((long long)(((h % 2046 + 1) << 52) | (mix(h) >> 12)));
    if (i % 4 == 1) y = 1.0 + (double)((int64_t)(h >> 12) - (int64_t)(1LL << 51)) * exp2(-52.0 - (double)(i % 50));
    if (i % 4 == 2) y = __longlong_as_double(0x3ff6a09e667f3bcdLL + (long long)(h % 4096) - 2048);
    if (i % 4 == 3) y = exp2((double)((int)(h % 2000) - 1000)) * (1.0 + (double)((int)((h >> 32) % 5) - 2) * 0x1p-52);
    check(bad, kLog, fast_log64(y), rg_log64(y), y, 0.0);
    const double any = __longlong_as_double((long long)mix(3 * i + 2));
    if (any == any) check(bad, kExact, halve(any), 0.5 * any, any, 0.0);
    check(bad, kExact, small_int((int)(h % 4096) - 2048), (double)((int)(h % 4096) - 2048), (double)i, 0.0);
    const double p = __longlong_as_double((long long)h);
    if (any == any && p == p) check(bad, kExact, order_key(any) < order_key(p), any < p, any, p);
  }
}

__global__ void normals(Bad* bad, uint64_t first, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(first + i);
    const double want = rg_probit64(((double)x + 0.5) * 0x1p-32);
    const bool tail = probit64_is_tail(x);
    const double got = tail ? probit64_tail(x) : probit64_central(x);
    if (__double_as_longlong(got) != __double_as_longlong(want) && atomicAdd(&bad->count[tail ? kTail : kCentral], 1ULL) == 0)
      bad->a[tail ? kTail : kCentral] = (double)x;
  }
}

int main() {
  Bad* bad = nullptr;
  if (cudaMalloc(&bad, sizeof(Bad)) != cudaSuccess || cudaMemset(bad, 0, sizeof(Bad)) != cudaSuccess) return 2;
  quotients<<<152 * 8, 256>>>(bad, 1ULL << 25);
  functions<<<152 * 8, 256>>>(bad, 1ULL << 26);
  for (uint64_t first = 0; first < (1ULL << 32); first += 1ULL << 28) normals<<<152 * 8, 256>>>(bad, first, 1ULL << 28);
  Bad h;
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(&h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) {
    std::printf("CUDA: %s\n", cudaGetErrorString(cudaGetLastError()));
    return 2;
  }
  const char* name[kChecks] = {"random quotients", "hardest quotients", "hardest quotients below two", "hardest quotients by a rounded reciprocal",
                               "exponential", "logarithm", "exact forms", "central inverse normals", "tail inverse normals"};
  int wrong = 0;
  for (int k = 0; k < kChecks; ++k) {
    std::printf("%s: %llu wrong", name[k], h.count[k]);
    if (h.count[k]) std::printf(" (%a, %a)", h.a[k], h.b[k]);
    std::printf("\n");
    wrong += h.count[k] != 0;
  }
  return wrong != 0;
}

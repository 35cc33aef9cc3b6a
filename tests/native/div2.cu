// Compares the problem module's div2 with the division operator, bit for bit (a NaN
// for a NaN): every pair of special operands, and random quotients by class of
// operand.  Prints the number of quotients compared and of those that differ.
#include <cstdint>
#include <cstdio>

#include "problem_ch.cuh"

using namespace bsam;

__device__ uint64_t mix(uint64_t x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__device__ double make(uint64_t sign, int exponent, uint64_t fraction) {
  return __longlong_as_double((long long)((sign << 63) | ((uint64_t)(exponent + 1023) << 52) |
                                          (fraction & 0xfffffffffffffull)));
}

__device__ bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y) || (isnan(x) && isnan(y));
}

__device__ int differ(double a, double b, double d) {
  double qa, qb;
  div2(a, b, d, qa, qb);
  return !same(qa, a / d) + !same(qb, b / d);
}

// Significands: anything, few bits set or cleared at either end.
__device__ uint64_t significand(uint64_t r) {
  const uint64_t f = mix(r);
  const int n = (int)(mix(r + 1) % 53);
  switch (mix(r + 2) % 4) {
    case 0: return f;
    case 1: return f >> n;                                    // near 1
    case 2: return ~(f >> (12 + n % 52));                     // near 2
    default: return (f & 7) | ((mix(f) & 7) << 49);           // few bits at both ends
  }
}

__global__ void k_random(int cls, uint64_t n, unsigned long long* bad) {
  unsigned long long mine = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = mix(i * 16 + cls) ^ ((uint64_t)cls << 60);
    double a, b, d;
    auto exponent = [&](int k, int lo, int hi) {
      return lo + (int)(mix(r + k) % (uint64_t)(hi - lo + 1));
    };
    auto sign = [&](int k) { return mix(r + k) >> 63; };
    if (cls == 0) {  // any bits at all
      a = __longlong_as_double((long long)mix(r + 1));
      b = __longlong_as_double((long long)mix(r + 2));
      d = __longlong_as_double((long long)mix(r + 3));
    } else if (cls == 1) {  // the update's own range: determinants of 1 and above
      d = make(0, exponent(1, 0, 20), mix(r + 2));
      a = make(sign(3), exponent(4, -30, 30), mix(r + 5));
      b = make(sign(6), exponent(7, -60, 60), mix(r + 8));
    } else if (cls == 2) {  // significands near both ends, inside the range
      d = make(sign(1), exponent(2, -399, 399), significand(r + 3));
      a = make(sign(4), exponent(5, -399, 399), significand(r + 9));
      b = make(sign(6), exponent(7, -399, 399), significand(r + 13));
    } else if (cls == 3) {  // divisors within 2^-15 below a power of two
      d = make(sign(1), exponent(2, -10, 10), ~(mix(r + 3) >> (27 + mix(r + 4) % 37)));
      a = make(sign(5), exponent(6, -10, 10), mix(r + 7));
      b = make(sign(8), exponent(9, -10, 10), significand(r + 10));
    } else if (cls == 4) {  // exponents about the bounds of the range
      auto edge = [&](int k) { return (sign(k) ? 400 : -400) + exponent(k + 1, -2, 2); };
      d = make(sign(1), sign(2) ? edge(3) : exponent(5, -3, 3), significand(r + 6));
      a = make(sign(10), sign(11) ? edge(12) : exponent(14, -3, 3), significand(r + 15));
      b = make(sign(19), edge(20), significand(r + 22));
    } else {  // quotients next to midpoints: a = (m + 1/2 ulp) d, rounded
      d = make(0, 0, significand(r + 1));
      const double m = make(0, 0, mix(r + 5));
      a = __fma_rn(m, d, 0x1p-53 * d);
      b = __fma_rn(m, d, -0x1p-53 * d);
    }
    mine += differ(a, b, d);
  }
  if (mine) atomicAdd(bad, mine);
}

constexpr int SPECIALS = 40;
__global__ void k_special(const double* v, unsigned long long* bad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= SPECIALS * SPECIALS * SPECIALS) return;
  const int n = differ(v[t % SPECIALS], v[t / SPECIALS % SPECIALS], v[t / SPECIALS / SPECIALS]);
  if (n) atomicAdd(bad, (unsigned long long)n);
}

int main() {
  unsigned long long* bad;
  double* v;
  if (cudaMallocManaged(&bad, 8) != cudaSuccess ||
      cudaMallocManaged(&v, sizeof(double) * SPECIALS) != cudaSuccess)
    return 2;
  *bad = 0;
  const double half[SPECIALS / 2] = {
      0.0, 0x1p-1074, 0x1.8p-1060, 0x1p-1022, 0x0.fffffffffffffp-1022, 0x1.fffffffffffffp+1023,
      __builtin_inf(), __builtin_nan(""), 1.0, 0x1.fffffffffffffp+0, 0x1.ffffep+0,
      0x1.ffffdffffffffp+0, 0x1p-400, 0x1.fffffffffffffp-401, 0x1.fffffffffffffp+399, 0x1p+400,
      3.0, 0x1.0000000000001p+0, 0x1.ffffefffffff0p+399, 0x1p+1023};
  for (int k = 0; k < SPECIALS; ++k) v[k] = k < SPECIALS / 2 ? half[k] : -half[k - SPECIALS / 2];
  const int cases = SPECIALS * SPECIALS * SPECIALS;
  k_special<<<(cases + 255) / 256, 256>>>(v, bad);
  double compared = 2.0 * cases;
  for (int cls = 0; cls < 6; ++cls) {
    const uint64_t n = 1ull << 30;
    k_random<<<148 * 8, 256>>>(cls, n, bad);
    compared += 2.0 * (double)n;
  }
  if (cudaDeviceSynchronize() != cudaSuccess) return 3;
  std::printf("%.0f %llu\n", compared, *bad);
  return *bad != 0;
}

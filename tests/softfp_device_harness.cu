// The device branches of softfp.cuh: the largest relative error of the hardware
// estimates over all their arguments, and the integer operations against the device's
// IEEE operations.
#include "../geon_gb300/csrc/softfp.cuh"

using namespace geon;

// estimate 0: 1/x for every FP32 x in [1, 2]; 1: 1/sqrt(x) for every x in [1, 4]
__global__ void estimate_error(int estimate, uint32_t count, unsigned long long* worst) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint32_t x = 0x3f800000u + i;
  const double v = (double)__uint_as_float(x);
  const double r = (double)__uint_as_float(estimate ? sf::rsqrt_bits(x) : sf::rcp_bits(x));
  // r / exact - 1, for the root from its square (r^2 x = 1 + 2 e + e^2)
  const double e = estimate ? fabs(fma(r * r, v, -1.0)) * 0.5 : fabs(fma(r, v, -1.0));
  atomicMax(worst, (unsigned long long)__double_as_longlong(e));
}

__device__ uint64_t mix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// significands by pattern: random, power of two, all ones, just above, just below, short, a run of ones, one bit
__device__ double make(uint64_t seed, int pattern, int exponents) {
  const uint64_t all = ((uint64_t)1 << 52) - 1, r = mix(seed), s = mix(r);
  uint64_t m = r & all;
  switch (pattern) {
    case 1: m = 0; break;
    case 2: m = all; break;
    case 3: m = r & 7; break;
    case 4: m = all ^ (r & 15); break;
    case 5: m &= ~(((uint64_t)1 << 30) - 1); break;
    case 6: m = ((uint64_t)1 << (r % 52)) - 1; break;
    case 7: m = (uint64_t)1 << (r % 52); break;
    default: break;
  }
  const uint64_t e = 1023 - exponents / 2 + s % exponents;
  return __longlong_as_double((long long)((e << 52) | m | (s >> 63 << 63)));
}

__device__ int differ(double a, double b) { return sf::bits(a) != sf::bits(b) && !(a != a && b != b); }

__global__ void operations(int pattern, uint64_t n, unsigned long long* bad) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t seed = mix(i * 8 + pattern);
  const double b = make(seed, i & 1 ? pattern : 0, i % 5 ? 400 : 1200);
  const double a = make(seed + 1, i & 2 ? pattern : 0, i % 7 ? 400 : 1200);
  int wrong = differ(sf::div(a, b), a / b) + differ(sf::rcp(b), 1.0 / b) + differ(sf::root(a), sqrt(a)) +
              differ(sf::root(fabs(a)), sqrt(fabs(a))) + differ(sf::half(a), 0.5 * a);
  // next to exact quotients and squares
  const double p = a * b, q = fabs(a) * fabs(a);
  const double pp = __longlong_as_double(__double_as_longlong(p) + (long long)(mix(seed + 2) % 3) - 1);
  const double qq = __longlong_as_double(__double_as_longlong(q) + (long long)(mix(seed + 3) % 5) - 2);
  wrong += differ(sf::div(pp, b), pp / b) + differ(sf::root(qq), sqrt(qq));
  wrong += isfinite(p) && fabs(p) >= 0x1p-1022 && differ(sf::mul(a, b), p);
  const double c = make(seed + 4, pattern, 338), d = make(seed + 5, i & 4 ? pattern : 0, 338);
  if (sf::spread(c) < sf::RANGE && sf::spread(d) < sf::RANGE) {
    wrong += differ(sf::mul(c, d), c * d) + differ(sf::mul(sf::mul(c, d), sf::mul(c, c)), (c * d) * (c * c)) +
             differ(sf::div_inside(c, d), c / d) + differ(sf::rcp_inside(d), 1.0 / d) +
             differ(sf::half_inside(c), 0.5 * c) + differ(sf::minus_twice_inside(c), -2.0 * c);
  }
  const uint64_t u = mix(seed + 6) >> 11 >> (mix(seed + 7) % 53);
  wrong += sf::unit53(u) != (double)u * 0x1p-53;
  if (wrong) atomicAdd(bad, (unsigned long long)wrong);
}

static unsigned long long result(unsigned long long* d) {
  unsigned long long h = ~0ull;
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) h = ~0ull;
  cudaFree(d);
  return h;
}

extern "C" double worst_estimate(int estimate) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 8) != cudaSuccess) return 1.0;
  cudaMemset(d, 0, 8);
  const uint32_t count = (estimate ? 2u << 23 : 1u << 23) + 1;
  estimate_error<<<(count + 255) / 256, 256>>>(estimate, count, d);
  const unsigned long long h = result(d);
  double e;
  memcpy(&e, &h, 8);
  return e;
}

extern "C" unsigned long long wrong_operations(int pattern, unsigned long long n) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 8) != cudaSuccess) return ~0ull;
  cudaMemset(d, 0, 8);
  operations<<<(unsigned)((n + 255) / 256), 256>>>(pattern, n, d);
  return result(d);
}

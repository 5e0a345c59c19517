// Compares the integer operations of softfp.cuh with the host's IEEE operations, bit for bit; prints the number of differences.
// argv: pattern of the significands (0-7), random cases, shift of the estimates
// in units in the last place.
#include <stdio.h>
#include <stdlib.h>

#include <random>

#include "../geon_gb300/csrc/softfp.cuh"

using namespace geon;

static std::mt19937_64 rng;

static double make(int pattern, int exponents) {
  const uint64_t all = ((uint64_t)1 << 52) - 1;
  uint64_t m = rng() & all;
  switch (pattern) {
    case 1: m = 0; break;                                   // powers of two
    case 2: m = all; break;                                 // all ones
    case 3: m = rng() & 7; break;                           // just above a power of two
    case 4: m = all ^ (rng() & 15); break;                  // just below one
    case 5: m &= ~(((uint64_t)1 << 30) - 1); break;         // short
    case 6: m = ((uint64_t)1 << (rng() % 52)) - 1; break;   // a run of ones
    case 7: m = (uint64_t)1 << (rng() % 52); break;         // one bit
    default: break;
  }
  const uint64_t e = 1023 - exponents / 2 + rng() % exponents;
  const uint64_t u = (e << 52) | m | ((rng() & 1) << 63);
  double x;
  memcpy(&x, &u, 8);
  return x;
}

static bool same(double a, double b) { return sf::bits(a) == sf::bits(b) || (a != a && b != b); }

int main(int argc, char** argv) {
  const int pattern = atoi(argv[1]);
  const long n = atol(argv[2]);
  sf::est_error() = atoi(argv[3]);
  rng.seed(977 + pattern);
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    const double b = make(i & 1 ? pattern : 0, i % 5 ? 400 : 1200), a = make(i & 2 ? pattern : 0, i % 7 ? 400 : 1200);
    bad += !same(sf::div(a, b), a / b);
    bad += !same(sf::rcp(b), 1.0 / b);
    bad += !same(sf::root(a), sqrt(a));
    bad += !same(sf::root(fabs(a)), sqrt(fabs(a)));
    // next to exact quotients and squares
    const double p = a * b, q = fabs(a) * fabs(a);  // (a b may leave the normal range)
    uint64_t up = sf::bits(p) + rng() % 3 - 1, uq = sf::bits(q) + rng() % 5 - 2;
    double pp, qq;
    memcpy(&pp, &up, 8);
    memcpy(&qq, &uq, 8);
    bad += !same(sf::div(pp, b), pp / b);
    bad += !same(sf::root(qq), sqrt(qq));
    bad += !same(sf::mul(a, b), p) && p - p == 0.0 && fabs(p) >= 0x1p-1022;
    const double c = make(pattern, 338), d = make(i & 4 ? pattern : 0, 338), e = make(0, 338);
    if (sf::spread(c) < sf::RANGE && sf::spread(d) < sf::RANGE && sf::spread(e) < sf::RANGE) {
      bad += !same(sf::mul(sf::mul(c, d), e), c * d * e) + !same(sf::mul(c, c), c * c);
      bad += !same(sf::mul(sf::mul(c, d), sf::mul(sf::mul(d, e), e)), (c * d) * ((d * e) * e));
    } else {
      ++bad;
    }
    bad += sf::half(a) != 0.5 * a;
    bad += sf::half_inside(c) != 0.5 * c || sf::half_inside(0.0) != 0.0 || sf::minus_twice_inside(c) != -2.0 * c;
    const uint64_t u = rng() >> 11 >> (rng() % 53);
    bad += sf::unit53(u) != (double)u * 0x1p-53;
    bad += sf::finite(pp) != (pp - pp == 0.0);
    bad += sf::below(a, 1e-8) != (fabs(a) < 1e-8);
  }
  const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, 2.2250738585072014e-308, 1e-310,
                            1.7e308, -1e308, 3.0, 0x1p-255, 0x1.fffffffffffffp-256, 0x1p257, 0x1.fffffffffffffp256, 0x1p-170, 0x1.fffffffffffffp-171, 0x1p170, 0x1.fffffffffffffp169,
                            1e-8, 0x1.5798ee2308c39p-27};
  for (double a : special) {
    bad += !same(sf::half(a), 0.5 * a);
    const double m = fabs(a);
    bad += (sf::spread(a) < sf::RANGE) != (m >= 0x1p-170 && m < 0x1p170);
    bad += !same(sf::root(a), sqrt(a)) + !same(sf::rcp(a), 1.0 / a);
    bad += sf::finite(a) != (a - a == 0.0);
    bad += sf::below(a, 1e-8) != (fabs(a) < 1e-8);
    for (double b : special) bad += !same(sf::div(a, b), a / b);
  }
  printf("%ld\n", bad);
  return 0;
}

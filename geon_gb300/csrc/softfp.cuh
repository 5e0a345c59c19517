// Correctly rounded FP64 division, reciprocal and square root in 32-bit integer
// arithmetic.
//
// GB300 executes FP64 at 1/64 of its integer and FP32 rate: a warp holds the
// FP64 pipe of an SM for 16-19 cycles per DADD, DMUL, DFMA or DSETP, and an
// IEEE division for 141 (square root 143, reciprocal 86; a division whose
// numerator is zero takes the slow path: 350), measured with independent
// chains at 16 warps per SM. The integer pipes of the same kernels are idle.
// The functions here return the same bits as the IEEE operations in 29 (div),
// 32 (root) and 27 (rcp) cycles that leave the FP64 pipe free, by digit
// recurrence on the 53-bit significands:
//   * a digit is the remainder's leading word times a hardware FP32 reciprocal
//     (or reciprocal square root) of the divisor, ~22 bits at a time; the
//     remainder after each digit is formed exactly (modulo 2^64, which holds it);
//   * after three digits the quotient (root) is known to within one unit and
//     its remainder is exact, so comparing twice the remainder with the divisor
//     (the remainder with the root) rounds to nearest. Neither a quotient nor a
//     root of FP64 numbers can be a tie.
// Digit recurrence with a reciprocal estimate: M. Ercegovac, T. Lang, "Division
// and Square Root: Digit-Recurrence Algorithms and Implementations" (1994),
// very-high-radix division by prescaling; the error bounds are beside the code.
// Operands outside [2^-255, 2^257) (zero, subnormal, huge, infinite, NaN) go to
// the hardware operation; a zero numerator is answered directly.
//
// Host and device code: the CPU tests compile it with g++ and compare it with
// the host's division and square root, moving the estimates by their error.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define GEON_SF __device__ __forceinline__
#else
#define GEON_SF inline
#endif

namespace geon {
namespace sf {

GEON_SF uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
GEON_SF double from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
GEON_SF uint32_t hi_of(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(x);
#else
  return (uint32_t)(bits(x) >> 32);
#endif
}
GEON_SF uint32_t lo_of(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(x);
#else
  return (uint32_t)bits(x);
#endif
}

// x is neither infinite nor NaN, without a DSETP
GEON_SF bool finite(double x) { return (hi_of(x) & 0x7ff00000u) != 0x7ff00000u; }

// |x| < t for a positive t (false for NaN): magnitudes order like their bits
GEON_SF bool below(double x, double t) { return (bits(x) & 0x7fffffffffffffffull) < bits(t); }

// 0.5 * x by its exponent
GEON_SF double half(double x) {
  const uint32_t h = hi_of(x), l = lo_of(x), e = h & 0x7ff00000u;
  if (e - 0x00200000u < 0x7fd00000u) return from_words(h - 0x00100000u, l);  // normal, and so is the half
  if (((h << 1) | l) == 0u) return x;
  return 0.5 * x;
}

// 0.5 * x for x zero or in [2^-1000, inf): no branch
GEON_SF double half_inside(double x) {
  const uint32_t h = hi_of(x), l = lo_of(x);
  return from_words(((h << 1) | l) ? h - 0x00100000u : h, l);
}

// -2 * x for a normal x whose double is finite: no branch
GEON_SF double minus_twice_inside(double x) { return from_words((hi_of(x) ^ 0x80000000u) + 0x00100000u, lo_of(x)); }

// (double)v * 2^-53 for v < 2^53 (exact)
GEON_SF double unit53(uint64_t v) {
  if (v == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int z = __clzll((long long)v);
#else
  const int z = __builtin_clzll(v);
#endif
  const uint64_t m = v << (z - 11);  // leading bit at 2^52
  return from_words((uint32_t)(m >> 32) + ((uint32_t)(1032 - z) << 20), (uint32_t)m);
}

// Estimates of 1/x (x in [1, 2]) and 1/sqrt(x) (x in [1, 4]) as FP32 bits (PTX
// rcp.approx, rsqrt.approx). What follows holds for relative errors up to RCP_ERROR
// (2^-22) and RSQRT_ERROR (2^-22.4); the hardware's are 2^-23.28 and 2^-22.94 at
// most, which a test measures over all these arguments. On the host the tests move
// the estimates, by units in the last place or by a part of those errors.
constexpr double RCP_ERROR = 0x1p-22, RSQRT_ERROR = 0x1.8p-23;
#ifdef __CUDA_ARCH__
GEON_SF uint32_t rcp_bits(uint32_t x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(x)));
  return __float_as_uint(r);
}
GEON_SF uint32_t rsqrt_bits(uint32_t x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(x)));
  return __float_as_uint(r);
}
GEON_SF uint32_t umulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
GEON_SF int32_t smulhi(int32_t a, int32_t b) { return __mulhi(a, b); }
#else
inline int& est_error() {
  static int e = 0;
  return e;
}
inline double& est_relative() {  // as a part of the bound, -1 to 1
  static double e = 0.0;
  return e;
}
// the FP32 number next to v (1 + e) on v's side (e = 0: nearest to v), moved by units
inline uint32_t moved(double v, double e) {
  const double w = v * (1.0 + e);
  float r = (float)w;
  if (e > 0.0 && (double)r > w) r = nextafterf(r, 0.0f);
  if (e < 0.0 && (double)r < w) r = nextafterf(r, 2.0f);
  uint32_t u;
  memcpy(&u, &r, 4);
  return u + est_error();
}
inline uint32_t rcp_bits(uint32_t x) {
  float f;
  memcpy(&f, &x, 4);
  return moved(1.0 / (double)f, RCP_ERROR * est_relative());
}
inline uint32_t rsqrt_bits(uint32_t x) {
  float f;
  memcpy(&f, &x, 4);
  return moved(1.0 / sqrt((double)f), RSQRT_ERROR * est_relative());
}
inline uint32_t umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int32_t smulhi(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
#endif

// Zero exactly when |x| (its high word) is in [2^-255, 2^257), else not zero.
GEON_SF uint32_t outside(uint32_t hi) { return (hi * 2u + 0xA0000000u) & 0xC0000000u; }

GEON_SF uint64_t pack(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// n - d * b modulo 2^64, d signed
GEON_SF uint64_t minus_product(uint64_t n, int32_t d, uint64_t b) {
  const uint32_t nd = (uint32_t)-d;
  uint64_t r = n + (uint64_t)nd * (uint32_t)b;
  uint32_t h = (uint32_t)(r >> 32) + nd * (uint32_t)(b >> 32);
  if (nd >> 31) h -= (uint32_t)b;  // nd as a signed factor
  return pack(h, (uint32_t)r);
}

// An FP32 estimate in [0.5, 1) as 2^31 times its value (ends clamped).
GEON_SF uint32_t fixed31(uint32_t r) {
  r = r > 0x3f000000u ? r : 0x3f000000u;
  r = r < 0x3f7fffffu ? r : 0x3f7fffffu;
  return ((r << 7) & 0x3fffffffu) | 0x40000000u;
}

// Significand (53 bits) of a / b rounded to nearest, for significands A' in
// [B, 2B) and B in [2^52, 2^53). Y = 2^31 times an estimate of 2^52 / B with
// relative error e at most 2^-21.67 (the estimate's RCP_ERROR = 2^-22 and its
// argument's 2^-24; the clamp moves a value beyond an end of [1/2, 1) to the end or,
// for B = 2^52, from 1 by 2^-24).
//   d1 ~ (A'/B) 2^30 < 2^31: error < 2^9.33 + 2  =>  |R1| < 2^9.4 B < 2^62.4
//   d2 ~ R1/B 2^19, |d2| < 2^28.4: error < 2^6.73 + 2  =>  |R2| < 2^6.8 B
//   d3 ~ floor(R2/B 2^3): error in [0, 1] and a part in 2^11 either way, so the
// quotient is Q = d1 2^22 + d2 2^3 + d3 plus R3 / B with R3 in (-B/2^11, 1.01 B).
GEON_SF uint64_t quotient(uint64_t A, uint64_t B, uint32_t Y) {
  const uint32_t d1 = umulhi((uint32_t)(A >> 22), Y << 1);
  uint64_t R = (A << 30) - ((uint64_t)d1 * (uint32_t)B + ((uint64_t)(d1 * (uint32_t)(B >> 32)) << 32));
  const int32_t d2 = smulhi((int32_t)(R >> 32), (int32_t)Y);
  R = minus_product(R << 19, d2, B);
  const int32_t d3 = smulhi((int32_t)(R >> 32), (int32_t)Y) >> 16;
  R = minus_product(R << 3, d3, B);
  uint64_t Q = ((uint64_t)d1 << 22) + (uint64_t)((int64_t)d2 * 8 + d3);
  if ((int64_t)(2 * R - B) > 0) ++Q;  // 2 R3 > B
  return Q;
}

// 2^31 times the estimate of 2^52 / B (the argument rounded to 24 bits).
GEON_SF uint32_t reciprocal_estimate(uint64_t B) {
  const uint32_t f = 0x3f800000u + ((uint32_t)((B + (1u << 28)) >> 29) - (1u << 23));
  return fixed31(rcp_bits(f));
}

// a / b for operands in [2^-255, 2^257)
GEON_SF double div_inside(double a, double b) {
  const uint32_t ah = hi_of(a), al = lo_of(a), bh = hi_of(b), bl = lo_of(b);
  const uint32_t am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
  const uint64_t B = pack(bm, bl);
  uint64_t A = pack(am, al);
  const uint32_t less = A < B ? 1u : 0u;
  A <<= less;
  const uint64_t Q = quotient(A, B, reciprocal_estimate(B));
  // exponents and signs: (ah - am) and (bh - bm) hold sign, exponent - 1
  const uint32_t h = (uint32_t)(Q >> 32) + (ah - am) - (bh - bm) + (1022u << 20) - (less << 20);
  return from_words(h, (uint32_t)Q);
}

// a / b, rounded to nearest: the bits of the IEEE division.
GEON_SF double div(double a, double b) {
  const uint32_t ah = hi_of(a), bh = hi_of(b);
  if (outside(bh) | outside(ah)) {
    if ((((ah << 1) | lo_of(a)) | outside(bh)) == 0u) return from_words((ah ^ bh) & 0x80000000u, 0u);  // +-0 / b
    return a / b;
  }
  return div_inside(a, b);
}

// 1 / b for b in [2^-255, 2^257)
GEON_SF double rcp_inside(double b) {
  const uint32_t bh = hi_of(b), bl = lo_of(b);
  const uint32_t bm = (bh & 0xfffffu) | 0x100000u;
  const uint64_t B = pack(bm, bl);
  const uint32_t less = (bl | (bm ^ 0x100000u)) ? 1u : 0u;  // B is not a power of two
  const uint64_t Q = quotient((uint64_t)1 << (52 + less), B, reciprocal_estimate(B));
  const uint32_t h = (uint32_t)(Q >> 32) + (1022u << 20) - (bh - bm) + (1022u << 20) - (less << 20);
  return from_words(h, (uint32_t)Q);
}

// 1 / b
GEON_SF double rcp(double b) { return outside(hi_of(b)) ? 1.0 / b : rcp_inside(b); }

// sqrt(a), rounded to nearest: the bits of the IEEE square root. With n in
// [1, 4) the significand (times 2 for an odd exponent), A = n 2^52, and y the
// estimate of 1/sqrt(n) (relative error at most RSQRT_ERROR = 2^-22.4, and half its
// argument's 2^-23: together 2^-22; the clamp only brings a value nearer, or moves
// 1 by 2^-24), Y = 2^31 y:
//   S1 ~ sqrt(n) 2^30: error < 2^9.1, R1 = n 2^60 - S1^2, |R1| < 2^41.1
//   d2 ~ R1 y 2^-12 (half the remainder over the root, 2^19 times finer):
//     T = S1 2^19 + d2 ~ sqrt(n) 2^49: error < 2^7.3, R2 = n 2^98 - T^2, |R2| < 2^58.3
//   d3 = floor(R2 y 2^-47): S = 2^3 T + d3, so sqrt(n) 2^52 lies in
//     [S, S + 1] and a part in 2^10 either way; it rounds up when its remainder
//     N - S^2 (N = n 2^104) exceeds S.
GEON_SF double root(double a) {
  const uint32_t ah = hi_of(a), al = lo_of(a);
  if (outside(ah) | (ah >> 31)) {
    return sqrt(a);
  }
  const uint32_t am = (ah & 0xfffffu) | 0x100000u;
  const uint32_t odd = ((ah >> 20) & 1u) ^ 1u;  // the unbiased exponent is odd
  const uint64_t A = pack(am, al) << odd;
  // n to 24 bits as FP32
  const uint32_t fb = 0x3f000000u + (odd << 23) + (uint32_t)(pack(am, al) >> 29);
  const uint32_t Y = fixed31(rsqrt_bits(fb));
  const uint32_t S1 = umulhi((uint32_t)(A >> 22), Y << 1);
  const uint64_t R1 = (A << 8) - (uint64_t)S1 * S1;
  const int32_t d2 = smulhi((int32_t)((int64_t)R1 >> 11), (int32_t)Y);
  const uint64_t T = ((uint64_t)S1 << 19) + (uint64_t)(int64_t)d2;
  const uint64_t R2 = minus_product(R1 << 38, d2, (T << 1) - (uint64_t)(int64_t)d2);
  const int32_t d3 = smulhi((int32_t)((int64_t)R2 >> 28), (int32_t)Y) >> 18;
  const uint64_t S = (T << 3) + (uint64_t)(int64_t)d3;
  // N - S^2 = R2 2^6 - d3 (2^4 T + d3)
  const uint64_t R3 = minus_product(R2 << 6, d3, (T << 4) + (uint64_t)(int64_t)d3);
  const uint64_t M = S + ((int64_t)(R3 - S) > 0 ? 1u : 0u);
  const uint32_t h = (uint32_t)(M >> 32) + ((((ah >> 20) - odd + 1021u) >> 1) << 20);
  return from_words(h, (uint32_t)M);
}

// How far |x| is from the middle of the range of mul's operands: below RANGE
// exactly when |x| is in [2^-170, 2^170). A kernel takes the largest over all
// operands it starts from and tests it once; products of up to six of them are
// then normal numbers, whatever the order.
constexpr uint32_t RANGE = 340u << 21;
GEON_SF uint32_t spread(double x) { return hi_of(x) * 2u - ((1023u - 170u) << 21); }

// a * b, rounded to nearest even, for normal operands whose product is normal:
// the bits of the IEEE multiplication in 15 cycles of the integer pipes (the
// FP64 pipe takes 19; sharing the multiplications between both brings a
// multiplication to 9.6). The significands are multiplied exactly in 32-bit
// pieces, a's moved up 11 bits so that the leading word of the product is the
// result's significand or half of it; the words below it round.
GEON_SF double mul(double a, double b) {
  const uint32_t ah = hi_of(a), al = lo_of(a), bh = hi_of(b), bl = lo_of(b);
  const uint32_t am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
  const uint64_t A = pack(am, al) << 11;
  const uint32_t A1 = (uint32_t)(A >> 32), A0 = (uint32_t)A;
  const uint64_t ll = (uint64_t)A0 * bl;
  const uint64_t m1 = (uint64_t)A1 * bl + (uint32_t)(ll >> 32);
  const uint64_t m2 = (uint64_t)A0 * bm + (uint32_t)m1;
  const uint64_t hh = (uint64_t)A1 * bm + ((uint64_t)(uint32_t)(m1 >> 32) + (uint32_t)(m2 >> 32));
  const uint32_t h1 = (uint32_t)(hh >> 32), w = (uint32_t)m2;
  const uint32_t sh = ((h1 >> 20) & 1u) ^ 1u;  // the product's significand is below 2
#ifdef __CUDA_ARCH__
  const uint64_t top = pack(__funnelshift_l((uint32_t)hh, h1, sh), __funnelshift_l(w, (uint32_t)hh, sh));
#else
  const uint64_t top = sh ? (hh << 1) | (w >> 31) : hh;
#endif
  // what is below, its last bit sticky: half or more rounds up, exactly half to even
  const uint32_t below_top = (w << sh) | ((uint32_t)ll ? 1u : 0u);
  const uint64_t carry = (uint64_t)below_top + (0x7fffffffu + ((uint32_t)top & 1u));
  const uint64_t m = top + (carry >> 32);
  const uint32_t h = (uint32_t)(m >> 32) + (ah - am) + (bh - bm) - (1021u << 20) - (sh << 20);
  return from_words(h, (uint32_t)m);
}

}  // namespace sf
}  // namespace geon

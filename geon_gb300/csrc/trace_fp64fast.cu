// GEON_FP64_FAST: an FP64 RK4 trace held to the tolerance of the reference's
// own CUDA kernel (cuda/schwarzschild_render.cu:3-5, "up to associativity")
// instead of to the reference's bits.
//
// Same chart, same fixed-step classical RK4 with the same stage points, the
// same termination tests (schwarzschild.rs:109-121) before every step and the
// same NaN guard and step cap (geodesic.rs:73-116) as the FP64 parity path, so
// a ray's class and final state differ from the reference only by rounding
// (amplified, as for any two FP64 evaluations, near the photon sphere). What is
// cheaper, per right-hand side (schwarzschild.rs:61-107 fused with
// geodesic.rs:38-59):
//   * one reciprocal, of D = r (r - 2M) sin(theta), in place of the reference's
//     five divisions: 1/r, Gamma^t_tr = M / (r (r - 2M)) and cot(theta) are
//     products with 1/D, and Gamma^r_tt = Gamma^t_tr f^2 with f = 1 - 2M/r;
//   * sin and cos of the polar angle carried from step to step: the three
//     later stages move theta by d = c h k^theta and take sin, cos of
//     theta0 + d by the angle-addition formula with Taylor polynomials of sin d
//     and cos d (|d| <= 1/32, truncation below 1e-19; larger offsets evaluate
//     sincos_det of the stage angle itself), the next step's theta0 the same
//     way from the step's own increment, and sincos_det afresh every 16 steps
//     of a ray (at load and after each group of 16 steps), so the carried
//     values stay within a few ulp;
//   * the sparse sums with fused multiply-adds, the Christoffel symbols shared
//     between their symmetric entries, and no stage positions for t and phi
//     (nothing reads them);
//   * multiplications, reciprocals and tests in the integer pipes (softfp.cuh),
//     beside the fused multiply-adds on the FP64 pipe;
//   * equatorial rays (bin/validate_shadow.rs:20-35: theta = pi/2, p^theta = 0)
//     step on their invariant plane with no trigonometry at all.
// Metrics other than Schwarzschild and Minkowski run the FP64 parity stepper
// (their Christoffel symbols come from the finite-difference fallback, whose
// cost is the metric evaluations, not the combination).
//
// This unit is compiled with --fmad=false like the others: every fused
// multiply-add below is written out.
#include <cuda_runtime.h>

#include "internal.h"
#include "metric_fp64.cuh"
#include "trace_common.cuh"

namespace geon {

namespace fast {

// Multiplication on the FP64 pipe or (SOFT) in the integer pipes, the same bits.
template <bool SOFT>
__device__ __forceinline__ double mul(double a, double b) {
  return SOFT ? sf::mul(a, b) : a * b;
}
// 1/x, correctly rounded, in the integer pipes
template <bool SOFT>
__device__ __forceinline__ double rcp(double x) {
  return SOFT ? sf::rcp_inside(x) : sf::rcp(x);
}
// -2 x
template <bool SOFT>
__device__ __forceinline__ double minus_twice(double x) {
  return SOFT ? sf::minus_twice_inside(x) : -2.0 * x;
}
// The largest sf::spread of the operands a soft step starts from.
struct Spread {
  uint32_t worst = 0;
  __device__ __forceinline__ void operator()(double x) {
    const uint32_t d = sf::spread(x);
    worst = d > worst ? d : worst;
  }
};

// sin(theta0 + d), cos(theta0 + d) from s0 = sin(theta0), c0 = cos(theta0) for
// |d| <= 1/32: sin d = d (1 - d^2/3! + d^4/5! - d^6/7!) (next term d^9/9! <
// 8e-20), cos d = 1 - d^2/2! + d^4/4! - d^6/6! + d^8/8! (next term < 3e-20).
template <bool SOFT>
__device__ __forceinline__ void sincos_offset(double s0, double c0, double d, double* s, double* c) {
  const double z = mul<SOFT>(d, d);
  double ps = fma(z, -1.0 / 5040.0, 1.0 / 120.0);
  ps = fma(z, ps, -1.0 / 6.0);
  const double sd = fma(mul<SOFT>(d, z), ps, d);
  double pc = fma(z, 1.0 / 40320.0, -1.0 / 720.0);
  pc = fma(z, pc, 1.0 / 24.0);
  pc = fma(z, pc, -0.5);
  const double cm1 = mul<SOFT>(z, pc);  // cos d - 1
  *s = fma(s0, cm1, fma(c0, sd, s0));
  *c = fma(c0, cm1, fma(-s0, sd, c0));
}

// Momentum derivatives of the Schwarzschild geodesic equation at radius r,
// polar angle with sin s and cos c, momentum p (k4..k7 of geodesic.rs:49-57).
// The reference's guard (schwarzschild.rs:98-102): cot(theta) = 0 where
// |sin theta| < 1e-8 (not in a soft step).
template <bool SOFT>
__device__ __forceinline__ void rhs(Spread& check, double m, double two_m, double r, double s, double c, double p0,
                                    double p1, double p2, double p3, double* k4, double* k5, double* k6, double* k7) {
  auto mul = [](double a, double b) { return fast::mul<SOFT>(a, b); };
  const double rm = r - two_m;
  const bool pole = !SOFT && sf::below(s, 1e-8);
  const double se = pole ? 1.0 : s;
  const double rrm = mul(r, rm);
  const double D = mul(rrm, se);
  const double iD = rcp<SOFT>(D);
  const double iDs = mul(iD, se);          // 1 / (r (r - 2M))
  const double ir = mul(rm, iDs);          // 1 / r
  const double cot = pole ? 0.0 : mul(c, mul(rrm, iD));
  const double u = mul(m, iDs);            // Gamma^t_tr = M / (r^2 f) = -Gamma^r_rr
  const double f = mul(rm, ir);            // 1 - 2M/r
  const double grtt = mul(u, mul(f, f));   // Gamma^r_tt = M f / r^2 = Gamma^t_tr f^2
  const double p3sq = mul(p3, p3);
  const double q = fma(mul(s, s), p3sq, mul(p2, p2));  // p_theta^2 + sin^2 p_phi^2
  *k4 = mul(mul(minus_twice<SOFT>(u), p0), p1);        // -2 Gamma^t_tr p^t p^r
  *k5 = fma(rm, q, fma(u, mul(p1, p1), mul(-mul(grtt, p0), p0)));
  *k6 = fma(mul(s, c), p3sq, mul(mul(minus_twice<SOFT>(ir), p1), p2));
  const double w7 = fma(ir, p1, mul(cot, p2));
  *k7 = mul(minus_twice<SOFT>(p3), w7);
  if (SOFT) {
    const double all[13] = {r, rm, s, c, p0, p1, p2, p3, D, u, f, cot, w7};
#pragma unroll
    for (int i = 0; i < 13; ++i) check(all[i]);
  }
}

// The same on the equatorial plane (s = 1, c = 0, p^theta = 0).
template <bool SOFT>
__device__ __forceinline__ void rhs_planar(Spread& check, double m, double two_m, double r, double p0, double p1,
                                           double p3, double* k4, double* k5, double* k7) {
  auto mul = [](double a, double b) { return fast::mul<SOFT>(a, b); };
  const double rm = r - two_m;
  const double D = mul(r, rm);
  const double iD = rcp<SOFT>(D);
  const double ir = mul(rm, iD);
  const double u = mul(m, iD);
  const double f = mul(rm, ir);
  const double grtt = mul(u, mul(f, f));
  *k4 = mul(mul(minus_twice<SOFT>(u), p0), p1);
  *k5 = fma(rm, mul(p3, p3), fma(u, mul(p1, p1), mul(-mul(grtt, p0), p0)));
  *k7 = mul(minus_twice<SOFT>(p3), mul(ir, p1));
  if (SOFT) {
    const double all[8] = {r, rm, p0, p1, p3, D, u, f};
#pragma unroll
    for (int i = 0; i < 8; ++i) check(all[i]);
  }
}

}  // namespace fast

// PLANAR: every ray is equatorial (the shadow source). Otherwise a ray that
// starts on the equator with p^theta = 0 exactly (theta = pi/2 to the double,
// as equatorial rays and states turned into their orbit-plane frame are)
// takes the planar step too: the plane is invariant, and the general step
// would only add the ~1e-16 drift that cos(pi/2 rounded) gives theta.
template <bool PLANAR>
struct FastSchwStepper {
  double y[8];
  bool on_plane = PLANAR;
  // sin and cos of y[2] for the general step, carried from step to step by
  // the angle-addition formula and taken afresh every 16 steps of the ray (at
  // load and after each group of 16 steps)
  double sth = 0.0, cth = 1.0;
  bool plain = false;  // FP64-pipe steps to the end of the group of steps
  __device__ __forceinline__ void load(const TraceLaunch&, const double y0[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = y0[i];
    if (!PLANAR) {
      on_plane = y[2] == 1.5707963267948966 && y[6] == 0.0;
      if (!on_plane) dm::sincos_det(y[2], &sth, &cth);
    }
  }
  __device__ __forceinline__ void to_double(double out[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = y[i];
  }
  __device__ __forceinline__ int terminate(const TraceLaunch& L) const {
    return metric_terminate<KIND_SCHWARZSCHILD>(L.M, y);
  }

  // One step into yn (and the sin and cos of its theta). The stages run in a
  // loop, one copy of the right-hand side. SOFT: the multiplications and
  // reciprocals run in the integer pipes without tests; false when an operand
  // was outside their range, the step moved theta by more than 1/32 or a pole
  // was near: the results then mean nothing and the step is repeated without
  // SOFT. The same bits either way.
  template <bool SOFT>
  __device__ __forceinline__ bool planar_step(const TraceLaunch& L, double yn[8]) const {
    const double m = L.M.p[0], two_m = 2.0 * m;
    double k4, k5, k7, a0, a1, a3, a4, a5, a7;
    double p0 = y[4], p1 = y[5], p3 = y[7], r = y[1];
    fast::Spread check;
    if (SOFT) check(m);
#pragma unroll 1
    for (int st = 0;; ++st) {
      fast::rhs_planar<SOFT>(check, m, two_m, r, p0, p1, p3, &k4, &k5, &k7);
      if (st == 3) break;
      if (st == 0) {
        a0 = p0; a1 = p1; a3 = p3; a4 = k4; a5 = k5; a7 = k7;
      } else {
        a0 = fma(2.0, p0, a0);
        a1 = fma(2.0, p1, a1);
        a3 = fma(2.0, p3, a3);
        a4 = fma(2.0, k4, a4);
        a5 = fma(2.0, k5, a5);
        a7 = fma(2.0, k7, a7);
      }
      const double c = st < 2 ? L.half_step : L.step;
      r = fma(c, p1, y[1]);
      p0 = fma(c, k4, y[4]);
      p1 = fma(c, k5, y[5]);
      p3 = fma(c, k7, y[7]);
    }
    const double sx = L.sixth;
    yn[0] = fma(sx, a0 + p0, y[0]); yn[1] = fma(sx, a1 + p1, y[1]); yn[2] = y[2]; yn[3] = fma(sx, a3 + p3, y[3]);
    yn[4] = fma(sx, a4 + k4, y[4]); yn[5] = fma(sx, a5 + k5, y[5]); yn[6] = y[6]; yn[7] = fma(sx, a7 + k7, y[7]);
    return !SOFT || check.worst < sf::RANGE;
  }

  template <bool SOFT>
  __device__ __forceinline__ bool general_step(const TraceLaunch& L, double yn[8], double* sn, double* cn) const {
    const double m = L.M.p[0], two_m = 2.0 * m;
    double k4, k5, k6, k7, acc[8];
    double p0 = y[4], p1 = y[5], p2 = y[6], p3 = y[7], r = y[1], s = sth, cs = cth;
    fast::Spread check;
    bool small = true;
    if (SOFT) {
      check(m);
      check(L.half_step);
    }
#pragma unroll 1
    for (int st = 0;; ++st) {
      fast::rhs<SOFT>(check, m, two_m, r, s, cs, p0, p1, p2, p3, &k4, &k5, &k6, &k7);
      if (SOFT) small &= !sf::below(s, 1e-8);
      if (st == 3) break;
      const double k[8] = {p0, p1, p2, p3, k4, k5, k6, k7};
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = st == 0 ? k[i] : fma(2.0, k[i], acc[i]);
      const double c = st < 2 ? L.half_step : L.step;
      const double d = fast::mul<SOFT>(c, p2);
      r = fma(c, p1, y[1]);
      p0 = fma(c, k4, y[4]);
      p1 = fma(c, k5, y[5]);
      p2 = fma(c, k6, y[6]);
      p3 = fma(c, k7, y[7]);
      if (SOFT) {
        check(d);
        small &= sf::below(d, 0x1.0000000000001p-5);
        fast::sincos_offset<true>(sth, cth, d, &s, &cs);
      } else if (sf::below(d, 0x1.0000000000001p-5)) {
        fast::sincos_offset<false>(sth, cth, d, &s, &cs);
      } else {
        dm::sincos_det(y[2] + d, &s, &cs);
      }
    }
    const double last[8] = {p0, p1, p2, p3, k4, k5, k6, k7};
#pragma unroll
    for (int i = 0; i < 8; ++i) yn[i] = fma(L.sixth, acc[i] + last[i], y[i]);
    // sin and cos at the new theta from those at the old one (the difference of
    // two nearby doubles is exact)
    const double dth = yn[2] - y[2];
    if (SOFT) {
      check(dth);
      small &= sf::below(dth, 0x1.0000000000001p-5);
      fast::sincos_offset<true>(sth, cth, dth, sn, cn);
      return small && check.worst < sf::RANGE;
    }
    if (sf::below(dth, 0x1.0000000000001p-5)) fast::sincos_offset<false>(sth, cth, dth, sn, cn);
    else if (sf::finite(yn[2])) dm::sincos_det(yn[2], sn, cn);
    return true;
  }

  // Before a group of steps: what the state tells about the integer step. A ray with
  // a momentum outside its range (zero is: radial rays on the plane, meridional ones
  // off it, in every step), at a pole, or turning by more than 1/32 a step would make
  // its warp take both steps, so the warp takes the FP64-pipe step if one of its rays
  // has to (36001 meridional rays of 400 steps 11.0 -> 7.1 ms; 4.6 for rays in the
  // integer step).
  __device__ __forceinline__ void group_begin(const TraceLaunch& L) {
    fast::Spread check;
    check(L.M.p[0]);
    check(y[4]);
    check(y[5]);
    check(y[7]);
    if (PLANAR || on_plane) {
      plain = __any_sync(__activemask(), check.worst >= sf::RANGE);
    } else {
      check(L.half_step);
      check(y[6]);
      const bool turns = !sf::below(L.step * y[6], 0x1.0000000000001p-5);
      plain = __any_sync(__activemask(), check.worst >= sf::RANGE || turns || sf::below(sth, 1e-8));
    }
  }

  __device__ __forceinline__ int step(const TraceLaunch& L) {
    double yn[8];
    if (PLANAR || on_plane) {
      if (plain || !planar_step<true>(L, yn)) planar_step<false>(L, yn);
      // t and phi advance by sums of the stage values of p^t and p^phi, which
      // the momentum increments contain: the guard on r and the momenta covers
      // them, and a sink that reads neither (the shadow sink) drops them.
      if (!(sf::finite(yn[1]) && sf::finite(yn[4]) && sf::finite(yn[5]) && sf::finite(yn[7]))) return STEP_NONFINITE;
      y[0] = yn[0]; y[1] = yn[1]; y[3] = yn[3]; y[4] = yn[4]; y[5] = yn[5]; y[7] = yn[7];
      return STEP_OK;
    }
    double sn = sth, cn = cth;
    if (plain || !general_step<true>(L, yn, &sn, &cn)) general_step<false>(L, yn, &sn, &cn);
    bool fin = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) fin &= sf::finite(yn[i]);
    if (!fin) return STEP_NONFINITE;
    sth = sn;
    cth = cn;
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = yn[i];
    return STEP_OK;
  }
  static constexpr bool FAST = false;
  __device__ __forceinline__ void group_end(const TraceLaunch&) {
    if (!PLANAR && !on_plane) dm::sincos_det(y[2], &sth, &cth);
  }
  __device__ __forceinline__ void check_null(const TraceLaunch&, const double*) {}
  __device__ __forceinline__ void finish(const TraceLaunch&) {}
};

// Bound by the FP64 pipe: the soft step leaves ~130 of its 272 instructions
// there. 36001 rays escaping from r = 30M (h 0.05, escape 100M): 54.8 -> 31.4 ms.
// One-warp blocks as in trace_fp64.cu; 12 per SM (168 registers: at 128 the
// general step spills twice as much).
template <int SRC, int SINK>
__global__ void __launch_bounds__(FP64_BLOCK, 12) trace_fp64fast_kernel(const TraceLaunch L) {
  trace_loop<FastSchwStepper<SRC == SRC_EQUATORIAL>, KIND_SCHWARZSCHILD, SRC, SINK>(L);
}

template <int SRC, int SINK>
static cudaError_t launch_fast(const TraceLaunch& L, cudaStream_t s) {
  static int sms = 0, per_sm = 0;
  if (sms == 0) {
    int dev = 0, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, trace_fp64fast_kernel<SRC, SINK>, FP64_BLOCK, 0);
    per_sm = occ < 1 ? 1 : occ;
  }
  trace_fp64fast_kernel<SRC, SINK><<<fp64_grid(sms, per_sm, L.reserve_per_sm, L.n), FP64_BLOCK, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_trace_fp64fast(const TraceLaunch& L, int src, int sink, cudaStream_t s) {
  if (L.n <= 0) return cudaSuccess;
  if (L.M.kind != KIND_SCHWARZSCHILD) return launch_trace_fp64(L, src, sink, s);
  if (src == SRC_EQUATORIAL && sink == SINK_SHADOW) return launch_fast<SRC_EQUATORIAL, SINK_SHADOW>(L, s);
  if (src == SRC_EQUATORIAL && sink == SINK_TRACE) return launch_fast<SRC_EQUATORIAL, SINK_TRACE>(L, s);
  if (src == SRC_ARRAY && sink == SINK_TRACE) return launch_fast<SRC_ARRAY, SINK_TRACE>(L, s);
  if (src == SRC_CAMERA && sink == SINK_RENDER) return launch_fast<SRC_CAMERA, SINK_RENDER>(L, s);
  if (src == SRC_CAMERA && sink == SINK_TRACE) return launch_fast<SRC_CAMERA, SINK_TRACE>(L, s);
  return cudaErrorInvalidValue;
}

}  // namespace geon

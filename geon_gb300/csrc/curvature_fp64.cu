// FP64 curvature (curvature.rs:25-141): Riemann -> Ricci -> R -> Einstein ->
// T_mu_nu -> T(k, k), for batches of points.
//
// The reference differentiates the Christoffel symbols with a point-local
// central difference at x +- 1e-5 e_alpha (curvature.rs:25-46), so every point
// needs Gamma at x and its 8 stencil neighbours. A block handles PPB points;
// its threads first evaluate those Christoffel arrays into shared memory (the
// stencil "halo" lives there), then contract them. Two facts cut the work
// without changing a bit:
//  - where g does not depend on x^alpha (every metric here ignores t; the
//    Schwarzschild and Morris-Thorne metrics also ignore phi), Gamma at
//    x +- h e_alpha is Gamma at x bit for bit, since no operation reads x^alpha.
//    Those stencil slots are not evaluated; the difference reads the centre
//    twice, (G - G) / 2h, as the reference's does.
//  - for the metrics with a generated sparse Christoffel (Alcubierre,
//    Morris-Thorne) the finite differences inside Gamma evaluate g at the
//    stencil point +- h e_beta. Those positions repeat between stencil points
//    (x + h e_1 + h e_2 serves both Gamma(x + h e_1) and Gamma(x + h e_2); the
//    coordinates are formed by the same additions), so g is evaluated once per
//    distinct position (31 instead of 63 for Alcubierre) and each Gamma is
//    formed from those values by the same generated expressions.
// Riemann is formed once per point: the reference forms it twice inside
// einstein() (ricci and ricci_scalar each call riemann) and again for every k
// in nec_contraction(), but it is deterministic, so the bits are the same.
//
// Compiled with --fmad=false; results match the CPU oracle bit for bit.
#include <cuda_runtime.h>

#include <cstring>

#include "internal.h"
#include "metric_fp64.cuh"

namespace geon {

#include "curvature_sparse.cuh"

constexpr int CURV_PPB = 16;       // points per block
constexpr int CURV_THREADS = 128;
static_assert(CURV_PPB <= 32 && CURV_THREADS >= 32 + CURV_PPB, "the tetrads run on the second warp");

// Axes g depends on (bit a for x^a).
template <int K>
constexpr int stencil_mask() {
  return K == KIND_MINKOWSKI ? 0 : (K == KIND_SCHWARZSCHILD || K == KIND_MORRIS_THORNE) ? 0x6 : 0xE;
}

__host__ __device__ constexpr int popcount4(int m) { return (m & 1) + ((m >> 1) & 1) + ((m >> 2) & 1) + ((m >> 3) & 1); }

// Stencil of one point for metric K. Slots: 0 the point, 1 + 2 i + m the point
// shifted by +h (m = 0) or -h (m = 1) along the i-th axis g depends on.
// Positions (metrics with values-based Gamma): 0 the point; 1 + 2 i + m one
// shift; 1 + 2 k + 4 i + 2 m + n two shifts along axis i, (x +- h) +- h;
// 1 + 6 k + 4 pair(i, j) + 2 m + n one shift along axis i and one along axis
// j > i.
template <int K>
struct Stencil {
  static constexpr int mask = stencil_mask<K>();
  static constexpr int k = popcount4(mask);
  static constexpr int slots = 1 + 2 * k;
  static constexpr int positions = 1 + 4 * k + 2 * k * k;

  __device__ static __forceinline__ int axis(int i) {  // i-th axis in the mask
    int seen = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if ((mask >> a) & 1) {
        if (seen == i) return a;
        ++seen;
      }
    return 0;
  }
  // Slot holding Gamma at x + h e_mu (minus = 0) or x - h e_mu (minus = 1).
  __device__ static __forceinline__ int slot_for(int mu, int minus) {
    if (!((mask >> mu) & 1)) return 0;
    return 1 + 2 * popcount4(mask & ((1 << mu) - 1)) + minus;
  }
  __device__ static __forceinline__ double shift(double v, int minus) { return minus ? v - FD_H : v + FD_H; }
  // Coordinates of slot s, formed as the reference forms its stencil points.
  __device__ static __forceinline__ void slot_point(const double x[4], int s, double xs[4]) {
    xs[0] = x[0]; xs[1] = x[1]; xs[2] = x[2]; xs[3] = x[3];
    if (s > 0) {
      const int a = axis((s - 1) >> 1);
      xs[a] = shift(x[a], (s - 1) & 1);
    }
  }
  __device__ static __forceinline__ int pair_index(int i, int j) { return i * (2 * k - i - 1) / 2 + (j - i - 1); }
  // Coordinates of position q: the stencil point, then the shift of the
  // finite difference inside Gamma (metric/mod.rs:25-43).
  __device__ static __forceinline__ void position(const double x[4], int q, double xq[4]) {
    xq[0] = x[0]; xq[1] = x[1]; xq[2] = x[2]; xq[3] = x[3];
    if (q == 0) return;
    q -= 1;
    if (q < 2 * k) {
      const int a = axis(q >> 1);
      xq[a] = shift(x[a], q & 1);
      return;
    }
    q -= 2 * k;
    if (q < 4 * k) {
      const int a = axis(q >> 2);
      xq[a] = shift(shift(x[a], (q >> 1) & 1), q & 1);
      return;
    }
    q -= 4 * k;
    const int pr = q >> 2;
    int i = 0, j = 1;
    for (int ii = 0; ii < k; ++ii)
      for (int jj = ii + 1; jj < k; ++jj)
        if (pair_index(ii, jj) == pr) { i = ii; j = jj; }
    const int a = axis(i), b = axis(j);
    xq[a] = shift(x[a], (q >> 1) & 1);
    xq[b] = shift(x[b], q & 1);
  }
  // Position of the finite-difference input `tag` of slot s; tag 0 is the
  // stencil point itself, tag 1 + 2 i + n its shift along the i-th axis.
  __device__ static __forceinline__ int input_position(int s, int tag) {
    if (s == 0) return tag;
    if (tag == 0) return s;
    const int i = (s - 1) >> 1, m = (s - 1) & 1;
    const int j = (tag - 1) >> 1, n = (tag - 1) & 1;
    if (i == j) return 1 + 2 * k + 4 * i + 2 * m + n;
    if (i < j) return 1 + 6 * k + 4 * pair_index(i, j) + 2 * m + n;
    return 1 + 6 * k + 4 * pair_index(j, i) + 2 * n + m;
  }
};

// Metric values at one position and Gamma from a slot's values: the metrics
// with a generated values-based Christoffel.
template <int K>
struct ValuesGamma {
  static constexpr int nv = 0;
};
template <>
struct ValuesGamma<KIND_ALCUBIERRE> {
  static constexpr int nv = ALCUBIERRE_VALUES;
  __device__ static __forceinline__ void eval(const MetricDesc& M, const double x[4], double* v) {
    alc_g00_g01(M, x, v, v + 1);
  }
  __device__ static __forceinline__ bool gamma(const double* gv, double* G) { return christoffel_alcubierre_from(gv, G); }
};
template <>
struct ValuesGamma<KIND_MORRIS_THORNE> {
  static constexpr int nv = MORRIS_THORNE_VALUES;
  __device__ static __forceinline__ void eval(const MetricDesc& M, const double x[4], double* v) {
    mt_g22_g33(M, x, v, v + 1);
  }
  __device__ static __forceinline__ bool gamma(const double* gv, double* G) {
    return christoffel_morris_thorne_from(gv, G);
  }
};

template <int K>
constexpr size_t curv_smem_doubles() {
  return (size_t)CURV_PPB * Stencil<K>::slots * 64 + (size_t)CURV_PPB * Stencil<K>::positions * ValuesGamma<K>::nv +
         (size_t)CURV_PPB * 16;
}

// Point p of a grid job: index p = (iz * ny + iy) * nx + ix, coordinate
// x^i = lo_i + i_i * ((hi_i - lo_i) / (n_i - 1)) (endpoints included), x^0 = t.
__device__ __forceinline__ void grid_point(const GridDesc& G, int64_t p, double x[4]) {
  const int64_t ix = p % G.n[0];
  const int64_t iy = (p / G.n[0]) % G.n[1];
  const int64_t iz = p / (G.n[0] * G.n[1]);
  x[0] = G.t;
  x[1] = G.n[0] > 1 ? G.lo[0] + (double)ix * ((G.hi[0] - G.lo[0]) / (double)(G.n[0] - 1)) : G.lo[0];
  x[2] = G.n[1] > 1 ? G.lo[1] + (double)iy * ((G.hi[1] - G.lo[1]) / (double)(G.n[1] - 1)) : G.lo[1];
  x[3] = G.n[2] > 1 ? G.lo[2] + (double)iz * ((G.hi[2] - G.lo[2]) / (double)(G.n[2] - 1)) : G.lo[2];
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Static observer tetrad of a point (Gram-Schmidt against g, as camera.rs:47-97
// builds it): rows e_0..e_3, tet[4 a + mu]. Returns false where the point has no
// static observer (g_tt >= 0 or a failed Gram-Schmidt step).
__device__ __forceinline__ bool point_tetrad(const double g[16], double tet[16]) {
#pragma unroll
  for (int q = 0; q < 16; ++q) tet[q] = 0.0;
  bool ok = g[0] < 0.0;
  if (ok) {
    tet[0] = 1.0 / sqrt(-g[0]);
    for (int i = 0; i < 3 && ok; ++i) {
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      v[i + 1] = 1.0;
      for (int kk = 0; kk <= i; ++kk) {
        const double coeff = dot4(g, tet + 4 * kk, v) / dot4(g, tet + 4 * kk, tet + 4 * kk);
        for (int mu = 0; mu < 4; ++mu) v[mu] -= coeff * tet[4 * kk + mu];
      }
      const double n2 = dot4(g, v, v);
      ok = n2 > 0.0;
      const double nn = sqrt(n2);
      for (int mu = 0; mu < 4; ++mu) tet[4 * (i + 1) + mu] = v[mu] / nn;
    }
  }
  return ok;
}

// Null vector q of point p: k = e0 + n1 e1 + n2 e2 + n3 e3 in the point's static
// observer tetrad, with n uniform on the unit sphere from the counter-based
// stream splitmix64(seed ^ (p * nk + q)): z = 2 u1 - 1, phi = 2 pi u2. Where the
// point has no static observer (ok false) k is NaN. The tetrad does not depend
// on q, so a point's tetrad is built once and shared by its nk vectors.
__device__ __forceinline__ void point_null_vector(const double* tet, bool ok, uint64_t seed, int64_t p,
                                                  int64_t nk, int64_t q, double k[4]) {
  const uint64_t h = splitmix64(seed ^ (uint64_t)(p * nk + q));
  const uint64_t h2 = splitmix64(h);
  const double u1 = (double)(h >> 11) * 0x1p-53, u2 = (double)(h2 >> 11) * 0x1p-53;
  const double z = 2.0 * u1 - 1.0;
  const double rho = sqrt(fmax(0.0, 1.0 - z * z));
  double sp, cp;
  dm::sincos_det(6.283185307179586 * u2, &sp, &cp);
  const double n1 = rho * cp, n2v = rho * sp, n3 = z;
#pragma unroll
  for (int mu = 0; mu < 4; ++mu) k[mu] = tet[mu] + n1 * tet[4 + mu] + n2v * tet[8 + mu] + n3 * tet[12 + mu];
  if (!ok) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    k[0] = k[1] = k[2] = k[3] = nan;
  }
}

// what: 0 riemann(256) 1 ricci(16) 2 ricci_scalar(1) 3 einstein(16) 4 stress_energy(16) 5 nec(nk)
//       6 grid job: einstein (out, 16 per point; may be null) and nec (out2, nk per point)
//         against generated null vectors (written to kout when not null)
template <int K, bool GRID>
__global__ void __launch_bounds__(CURV_THREADS)
curvature_kernel(const MetricDesc M, int what, const double* __restrict__ xs, int64_t n,
                 const double* __restrict__ ks, int64_t nk, int k_shared, double* __restrict__ out,
                 int* flags, const GridDesc grid, uint64_t seed, double* __restrict__ out2,
                 double* __restrict__ kout) {
  using ST = Stencil<K>;
  using VG = ValuesGamma<K>;
  constexpr int NS = ST::slots, NP = ST::positions, NV = VG::nv;
  extern __shared__ double smem[];
  double* G = smem;                                     // [PPB][NS][64]
  double* PV = G + CURV_PPB * NS * 64;                  // [PPB][NP][NV]
  double* RIC = PV + CURV_PPB * NP * NV;                // [PPB][16]
  const int tid = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * CURV_PPB;
  auto point = [&](int64_t pt, double x[4]) {
    if (GRID) {
      grid_point(grid, pt, x);
    } else {
      x[0] = xs[4 * pt]; x[1] = xs[4 * pt + 1]; x[2] = xs[4 * pt + 2]; x[3] = xs[4 * pt + 3];
    }
  };

  // 1. Christoffel symbols at the stencil slots of each point.
  if constexpr (NV > 0) {
    for (int e = tid; e < CURV_PPB * NP; e += CURV_THREADS) {
      const int p = e / NP, q = e - NP * (e / NP);
      if (p0 + p >= n) continue;
      double x[4], xq[4];
      point(p0 + p, x);
      ST::position(x, q, xq);
      VG::eval(M, xq, PV + (p * NP + q) * NV);
    }
    __syncthreads();
    for (int e = tid; e < CURV_PPB * NS; e += CURV_THREADS) {
      const int p = e / NS, sl = e - NS * (e / NS);
      if (p0 + p >= n) continue;
      double gv[NS * NV];
#pragma unroll
      for (int tag = 0; tag < NS; ++tag) {
        const double* v = PV + (p * NP + ST::input_position(sl, tag)) * NV;
#pragma unroll
        for (int c = 0; c < NV; ++c) gv[tag * NV + c] = v[c];
      }
      if (!VG::gamma(gv, G + (p * NS + sl) * 64)) atomicOr(flags, 1);
    }
  } else {
    for (int e = tid; e < CURV_PPB * NS; e += CURV_THREADS) {
      const int p = e / NS, sl = e - NS * (e / NS);
      if (p0 + p >= n) continue;
      double x[4], xsl[4];
      point(p0 + p, x);
      ST::slot_point(x, sl, xsl);
      if (!metric_christoffel<K>(M, xsl, G + (p * NS + sl) * 64)) atomicOr(flags, 1);
    }
  }
  __syncthreads();

  const double inv_2h = 1.0 / (2.0 * FD_H);
  // Riemann entry R^rho_{sigma mu nu} (curvature.rs:48-70) from the shared stencil.
  auto riem = [&](int p, int rho, int sigma, int mu, int nu) -> double {
    const double* g0 = G + (p * NS) * 64;
    const double* gpm = G + (p * NS + ST::slot_for(mu, 0)) * 64;
    const double* gmm = G + (p * NS + ST::slot_for(mu, 1)) * 64;
    const double* gpn = G + (p * NS + ST::slot_for(nu, 0)) * 64;
    const double* gmn = G + (p * NS + ST::slot_for(nu, 1)) * 64;
    const double term1 = (gpm[16 * rho + 4 * nu + sigma] - gmm[16 * rho + 4 * nu + sigma]) * inv_2h;
    const double term2 = (gpn[16 * rho + 4 * mu + sigma] - gmn[16 * rho + 4 * mu + sigma]) * inv_2h;
    double term3 = 0.0, term4 = 0.0;
#pragma unroll
    for (int lambda = 0; lambda < 4; ++lambda) {
      term3 += g0[16 * rho + 4 * mu + lambda] * g0[16 * lambda + 4 * nu + sigma];
      term4 += g0[16 * rho + 4 * nu + lambda] * g0[16 * lambda + 4 * mu + sigma];
    }
    return term1 - term2 + term3 - term4;
  };

  if (what == 0) {
    for (int e = tid; e < CURV_PPB * 256; e += CURV_THREADS) {
      const int p = e >> 8, q = e & 255;
      const int64_t pt = p0 + p;
      if (pt >= n) continue;
      out[256 * pt + q] = riem(p, q >> 6, (q >> 4) & 3, (q >> 2) & 3, q & 3);
    }
    return;
  }

  // 2. Ricci R_mu_nu = sum_alpha R^alpha_{mu alpha nu} (curvature.rs:72-85).
  for (int e = tid; e < CURV_PPB * 16; e += CURV_THREADS) {
    const int p = e >> 4, mu = (e >> 2) & 3, nu = e & 3;
    if (p0 + p >= n) continue;
    double s = 0.0;
#pragma unroll
    for (int alpha = 0; alpha < 4; ++alpha) s += riem(p, alpha, mu, alpha, nu);
    RIC[16 * p + 4 * mu + nu] = s;
  }
  __syncthreads();

  // 3. One thread per point: R, G, T. Ricci, R, G and T end here.
  if (what <= 4) {
    if (tid >= CURV_PPB) return;
    const int p = tid;
    const int64_t pt = p0 + p;
    if (pt >= n) return;
    const double* ric = RIC + 16 * p;
    if (what == 1) {
      for (int q = 0; q < 16; ++q) out[16 * pt + q] = ric[q];
      return;
    }
    double x[4];
    point(pt, x);
    double g[16], gi[16];
    metric_g<K>(M, x, g);
    if (!metric_g_inv_given<K>(M, x, g, gi)) atomicOr(flags, 1);
    double rs = 0.0;  // curvature.rs:87-97
#pragma unroll
    for (int q = 0; q < 16; ++q) rs += gi[q] * ric[q];
    if (what == 2) {
      out[pt] = rs;
      return;
    }
    const double factor = 1.0 / (8.0 * 3.141592653589793);
    for (int q = 0; q < 16; ++q) {
      const double ein = ric[q] - 0.5 * g[q] * rs;             // curvature.rs:99-110
      out[16 * pt + q] = what == 3 ? ein : ein * factor;      // curvature.rs:112-122
    }
    return;
  }

  // what 5 and 6: T_mu_nu per point (written over the point's Ricci row), and
  // for the grid job the point's tetrad (over the first stencil slots: the
  // Christoffel arrays are no longer read).
  double* TT = RIC;
  double* TET = G;                                    // [PPB][16]
  int* TOK = (int*)(G + CURV_PPB * 16);               // [PPB]
  // The Einstein and stress-energy tensors on the first CURV_PPB threads and,
  // for the grid job, the tetrads on as many threads of the next warp (both
  // start from g of the point, evaluated on each side), so the block's serial
  // part is the longer of the two instead of their sum.
  if (tid < CURV_PPB && p0 + tid < n) {
    const int p = tid;
    const int64_t pt = p0 + p;
    double* ric = RIC + 16 * p;
    double x[4];
    point(pt, x);
    double g[16], gi[16];
    metric_g<K>(M, x, g);
    if (!metric_g_inv_given<K>(M, x, g, gi)) atomicOr(flags, 1);
    double rs = 0.0;  // curvature.rs:87-97
#pragma unroll
    for (int q = 0; q < 16; ++q) rs += gi[q] * ric[q];
    const double factor = 1.0 / (8.0 * 3.141592653589793);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const double ein = ric[q] - 0.5 * g[q] * rs;    // curvature.rs:99-110
      if (what == 6 && out) out[16 * pt + q] = ein;
      ric[q] = ein * factor;                           // curvature.rs:112-122
    }
  } else if (what == 6 && tid >= 32 && tid < 32 + CURV_PPB && p0 + (tid - 32) < n) {
    const int p = tid - 32;
    double x[4], g[16], tet[16];
    point(p0 + p, x);
    metric_g<K>(M, x, g);
    TOK[p] = point_tetrad(g, tet) ? 1 : 0;
#pragma unroll
    for (int q = 0; q < 16; ++q) TET[16 * p + q] = tet[q];
  }
  __syncthreads();

  // 4. T(k, k) (nec_contraction, curvature.rs:127-136), one (point, vector)
  // pair per thread.
  const int64_t pairs = (int64_t)CURV_PPB * nk;
  for (int64_t e = tid; e < pairs; e += CURV_THREADS) {
    const int p = (int)(e / nk);
    const int64_t c = e - (int64_t)p * nk;
    const int64_t pt = p0 + p;
    if (pt >= n) continue;
    const double* t = TT + 16 * p;
    double k[4];
    if (what == 6) {
      point_null_vector(TET + 16 * p, TOK[p] != 0, seed, pt, nk, c, k);
      if (kout)
        for (int mu = 0; mu < 4; ++mu) kout[4 * (pt * nk + c) + mu] = k[mu];
    } else {
      const double* kp = k_shared ? ks + 4 * c : ks + 4 * (pt * nk + c);
      k[0] = kp[0]; k[1] = kp[1]; k[2] = kp[2]; k[3] = kp[3];
    }
    double sacc = 0.0;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
#pragma unroll
      for (int nu = 0; nu < 4; ++nu) sacc += t[4 * mu + nu] * k[mu] * k[nu];
    (what == 6 ? out2 : out)[pt * nk + c] = sacc;
  }
}

// ---------------------------------------------------------------------------
// One thread per point (Alcubierre, Morris-Thorne, Schwarzschild).
//
// The cooperative kernel above spends most of its FP64 operations on structural
// zeros (dense Riemann sums, dense Gram-Schmidt) and leaves lanes idle in its
// per-point parts. Here a thread evaluates a whole point with the generated
// sparse code of curvature_sparse.cuh: the metric values of the stencil into
// shared memory (one column per thread), the distinct nonzero symbols slot by
// slot, their differences, the sparse Ricci tensor, and the vectors of the point
// one after another. Terms that are structurally zero, or the difference of two
// equal values, are left out. Such a term of the dense sums is a zero while
// nothing overflows, so results have the dense code's bits up to the sign of a
// zero where every symbol is below SYMBOL_BOUND; a point with a singular metric
// or a larger or non-finite symbol goes through the dense sums (dense_ricci),
// where 0 * inf and inf - inf are NaN as they are in the reference.
// Divisions and square roots run in the integer pipes (softfp.cuh), and so do
// the tests and the conversion of the random directions. Still bound by the FP64
// pipe, with about 4400 instead of 10400 FP64 operations per Alcubierre point
// and 32 of 32 lanes instead of 27: 128^3 points with 16 vectors 43.4 -> 18.2 ms,
// 32736 Morris-Thorne points 518 -> 170 us, 10^5 Schwarzschild scalars 486 -> 90 us.
// ---------------------------------------------------------------------------
constexpr int POINT_THREADS = 64;
// High word of 2^500. Below it products of two symbols stay below 2^1000, their
// differences over 2 h below 2^518, and the sums of a Riemann entry finite.
constexpr unsigned SYMBOL_BOUND = (1023u + 500u) << 20;

// Ricci tensor of one point by the dense sums of curvature.rs:48-85.
template <int K>
__device__ __noinline__ void dense_ricci(const MetricDesc& M, const double x[4], double* ric, int* flags) {
  using ST = Stencil<K>;
  double G[ST::slots][64];
  for (int sl = 0; sl < ST::slots; ++sl) {
    double xs[4];
    ST::slot_point(x, sl, xs);
    if (!metric_christoffel<K>(M, xs, G[sl])) atomicOr(flags, 1);
  }
  const double inv_2h = 1.0 / (2.0 * FD_H);
  for (int mu = 0; mu < 4; ++mu)
    for (int nu = 0; nu < 4; ++nu) {
      double s = 0.0;
      for (int al = 0; al < 4; ++al) {  // R^al_{mu al nu}
        const double* g0 = G[0];
        const double term1 = (G[ST::slot_for(al, 0)][16 * al + 4 * nu + mu] - G[ST::slot_for(al, 1)][16 * al + 4 * nu + mu]) * inv_2h;
        const double term2 = (G[ST::slot_for(nu, 0)][16 * al + 4 * al + mu] - G[ST::slot_for(nu, 1)][16 * al + 4 * al + mu]) * inv_2h;
        double term3 = 0.0, term4 = 0.0;
        for (int la = 0; la < 4; ++la) {
          term3 += g0[16 * al + 4 * al + la] * g0[16 * la + 4 * nu + mu];
          term4 += g0[16 * al + 4 * nu + la] * g0[16 * la + 4 * al + mu];
        }
        s += term1 - term2 + term3 - term4;
      }
      ric[4 * mu + nu] = s;
    }
}

// What the point kernel needs of a metric:
//   NV doubles of metric values per thread, ND differences per axis;
//   values(M, x, v): the metric values of every stencil position, v[q * THREADS];
//   symbols(M, x, v, slot, c): the distinct symbols of a slot;
//   ricci(c, d, ric), metric(M, x, v, g, gi): the nonzero entries of g and g^-1;
//   diff_place(i): the place of symbol i among the stored differences, or -1;
//   GMASK: the entries of g that are not zero.
template <int K>
struct PointMetric;

template <>
struct PointMetric<KIND_ALCUBIERRE> {
  using ST = Stencil<KIND_ALCUBIERRE>;
  static constexpr int NG = ALCUBIERRE_GAMMAS, ND = ALCUBIERRE_DIFFS, GMASK = 0x8433;
  // the metric function f at the 31 positions; while they are formed, the
  // squares of the 7 shifted coordinates per axis lie where the differences will
  static constexpr int NV = ST::positions;
  static_assert(21 <= 3 * ND, "the squares fit into the store of the differences");
  __device__ static __forceinline__ void values(const MetricDesc& M, const double x[4], double* v, double* store) {
    // shifts of one axis: 0, +h, -h, then (+h) +h, (+h) -h, (-h) +h, (-h) -h
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double c = x[a + 1], p = c + FD_H, m = c - FD_H;
      const double s[7] = {c, p, m, p + FD_H, p - FD_H, m + FD_H, m - FD_H};
#pragma unroll
      for (int i = 0; i < 7; ++i) {
        const double d = a == 0 ? s[i] - M.p[3] : s[i];
        store[(7 * a + i) * POINT_THREADS] = d * d;
      }
    }
    const double R = M.p[0], th = M.p[1];
#pragma unroll 1
    for (int q = 0; q < ST::positions; ++q) {  // Stencil::position's numbering
      int sx = 0, sy = 0, sz = 0;
      if (q >= 1 && q < 7) {
        const int a = (q - 1) >> 1, i = 1 + ((q - 1) & 1);
        sx = a == 0 ? i : 0, sy = a == 1 ? i : 0, sz = a == 2 ? i : 0;
      } else if (q >= 7 && q < 19) {
        const int a = (q - 7) >> 2, i = 3 + ((q - 7) & 3);
        sx = a == 0 ? i : 0, sy = a == 1 ? i : 0, sz = a == 2 ? i : 0;
      } else if (q >= 19) {
        const int pr = (q - 19) >> 2, i = 1 + (((q - 19) >> 1) & 1), j = 1 + ((q - 19) & 1);
        sx = pr < 2 ? i : 0, sy = pr == 0 ? j : (pr == 2 ? i : 0), sz = pr >= 1 ? j : 0;
      }
      const double rs = sf::root(store[sx * POINT_THREADS] + store[(7 + sy) * POINT_THREADS] +
                                 store[(14 + sz) * POINT_THREADS]);
      const double t_plus = dm::tanh_det(sf::div(rs + R, th));
      const double t_minus = dm::tanh_det(sf::div(rs - R, th));
      v[q * POINT_THREADS] = sf::div(t_plus - t_minus, M.alc_denom);
    }
  }
  __device__ static __forceinline__ void entry(const MetricDesc& M, double f, double* g00, double* g01) {
    const double v = M.p[2];
    *g00 = -1.0 + v * v * f * f;
    *g01 = -v * f;
  }
  __device__ static __forceinline__ bool symbols(const MetricDesc& M, const double*, const double* v, int slot, double* c) {
    double gv[14];
#pragma unroll
    for (int tag = 0; tag < 7; ++tag)
      entry(M, v[ST::input_position(slot, tag) * POINT_THREADS], gv + 2 * tag, gv + 2 * tag + 1);
    return alcubierre_gammas(gv, c);
  }
  template <class D>
  __device__ static __forceinline__ void ricci(const double* c, D d, double* ric) { alcubierre_ricci(c, d, ric); }
  __device__ static constexpr int diff_place(int i) { return alcubierre_diff_place(i); }
  __device__ static __forceinline__ void metric(const MetricDesc& M, const double*, const double* v, double* g, double* gi) {
    double gv[2];
    entry(M, v[0], gv, gv + 1);
    g[0] = gv[0]; g[1] = gv[1]; g[4] = gv[1]; g[5] = 1.0; g[10] = 1.0; g[15] = 1.0;
    alcubierre_inverse(gv, gi);
  }
};

template <>
struct PointMetric<KIND_MORRIS_THORNE> {
  using ST = Stencil<KIND_MORRIS_THORNE>;
  static constexpr int NG = MORRIS_THORNE_GAMMAS, ND = MORRIS_THORNE_DIFFS, GMASK = 0x8421;
  // r^2 = b0^2 + l^2 at the 7 shifted l and sin(theta) at the 7 shifted theta
  static constexpr int NV = 14;
  __device__ static __forceinline__ void values(const MetricDesc& M, const double x[4], double* v, double*) {
    const double b0 = M.p[0];
#pragma unroll 1
    for (int i = 0; i < 7; ++i) {
      const int s1 = i < 3 ? i : 1 + ((i - 3) >> 1), s2 = i < 3 ? 0 : 1 + ((i - 3) & 1);
      double l = x[1], th = x[2];
      if (s1) l = ST::shift(l, s1 - 1), th = ST::shift(th, s1 - 1);
      if (s2) l = ST::shift(l, s2 - 1), th = ST::shift(th, s2 - 1);
      v[i * POINT_THREADS] = b0 * b0 + l * l;
      double s, c;
      dm::sincos_det(th, &s, &c);
      v[(7 + i) * POINT_THREADS] = s;
    }
  }
  // g_thth and g_phph at shift i of l and shift j of theta (mt_g22_g33)
  __device__ static __forceinline__ void entry(const double* v, int i, int j, double* g) {
    const double r2 = v[i * POINT_THREADS], s = v[(7 + j) * POINT_THREADS];
    g[0] = r2;
    g[1] = r2 * s * s;
  }
  __device__ static __forceinline__ bool symbols(const MetricDesc&, const double*, const double* v, int slot, double* c) {
    // slot: 0 the point, 1 + m its shift along l, 3 + m along theta; tag 1 + n along l, 3 + n along theta
    const int li = slot == 1 || slot == 2 ? slot : 0, ti = slot >= 3 ? slot - 2 : 0;
    double gv[10];
    entry(v, li, ti, gv);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      entry(v, li ? 1 + 2 * li + n : 1 + n, ti, gv + 2 + 2 * n);
      entry(v, li, ti ? 1 + 2 * ti + n : 1 + n, gv + 6 + 2 * n);
    }
    return morris_thorne_gammas(gv, c);
  }
  template <class D>
  __device__ static __forceinline__ void ricci(const double* c, D d, double* ric) { morris_thorne_ricci(c, d, ric); }
  __device__ static constexpr int diff_place(int i) { return morris_thorne_diff_place(i); }
  __device__ static __forceinline__ void metric(const MetricDesc&, const double*, const double* v, double* g, double* gi) {
    double gv[2];
    entry(v, 0, 0, gv);
    g[0] = -1.0; g[5] = 1.0; g[10] = gv[0]; g[15] = gv[1];
    morris_thorne_inverse(gv, gi);
  }
};

template <>
struct PointMetric<KIND_SCHWARZSCHILD> {
  using ST = Stencil<KIND_SCHWARZSCHILD>;
  static constexpr int NG = 8, ND = SCHWARZSCHILD_DIFFS, GMASK = 0x8421;
  static constexpr int NV = 0;
  __device__ static __forceinline__ void values(const MetricDesc&, const double*, double*, double*) {}
  // christoffel_schw's entries: t_tr, r_tt, r_rr, r_thth, r_phph, 1/r, th_phph, cot
  __device__ static __forceinline__ bool symbols(const MetricDesc& M, const double* x, const double*, int slot, double* c) {
    double r = x[1], theta = x[2];
    const double m = M.p[0];
    if (slot == 1 || slot == 2) r = ST::shift(r, slot - 1);
    if (slot >= 3) theta = ST::shift(theta, slot - 3);
    const double f = 1.0 - sf::div(2.0 * m, r);
    double sin_t, cos_t;
    dm::sincos_det(theta, &sin_t, &cos_t);
    const double gtr = sf::div(m, r * r * f);
    c[0] = gtr;
    c[1] = sf::div(m * f, r * r);
    c[2] = -gtr;
    c[3] = -(r - 2.0 * m);
    c[4] = c[3] * sin_t * sin_t;
    c[5] = sf::rcp(r);
    c[6] = -sin_t * cos_t;
    c[7] = sf::below(sin_t, 1e-8) ? 0.0 : sf::div(cos_t, sin_t);
    return true;
  }
  template <class D>
  __device__ static __forceinline__ void ricci(const double* c, D d, double* ric) { schwarzschild_ricci(c, d, ric); }
  __device__ static constexpr int diff_place(int i) { return schwarzschild_diff_place(i); }
  __device__ static __forceinline__ void metric(const MetricDesc& M, const double* x, const double*, double* g, double* gi) {
    const double r = x[1], m = M.p[0];
    const double f = 1.0 - sf::div(2.0 * m, r);
    double sin_t, cos_t;
    dm::sincos_det(x[2], &sin_t, &cos_t);
    const double rr = r * r, rrss = rr * sin_t * sin_t;
    g[0] = -f; g[5] = sf::rcp(f); g[10] = rr; g[15] = rrss;
    gi[0] = -g[5]; gi[5] = f; gi[10] = sf::rcp(rr); gi[15] = sf::rcp(rrss);
  }
};

// T(k, k) of a point's generated vectors with the dense Gram-Schmidt and sums.
__device__ __noinline__ void dense_contractions(const double* g, const double* t, uint64_t seed, int64_t pt, int64_t nk,
                                                double* nec, double* kout) {
  double tet[16];
  const bool ok = point_tetrad(g, tet);
  for (int64_t q = 0; q < nk; ++q) {
    double k[4];
    point_null_vector(tet, ok, seed, pt, nk, q, k);
    double sacc = 0.0;
    for (int mu = 0; mu < 4; ++mu) {
      if (kout) kout[4 * (pt * nk + q) + mu] = k[mu];
      for (int nu = 0; nu < 4; ++nu) sacc += t[4 * mu + nu] * k[mu] * k[nu];
    }
    nec[pt * nk + q] = sacc;
  }
}

// The static observer's tetrad of a point (point_tetrad) with the zero terms of
// the Gram-Schmidt sums left out, for points whose symbols are below SYMBOL_BOUND
// (g is finite there; an infinite entry makes 0 * inf of the terms left out): e0 = a d_t, e1 = (b, c, 0, 0), e2 and e3 along
// their axes. Diagonal metrics have b = 0.
struct SparseTetrad {
  double a, b, c, e2, e3;
  bool ok;
};
template <int K>
__device__ __forceinline__ SparseTetrad sparse_tetrad(const double* g) {
  SparseTetrad t;
  const double a = sf::rcp(sf::root(-g[0]));
  t.a = a;
  t.ok = g[0] < 0.0;
  if (K == KIND_ALCUBIERRE) {
    const double coeff = sf::div(g[1] * a, g[0] * a * a);
    const double v0 = 0.0 - coeff * a;
    const double n2 = plus_zero(g[0] * v0 * v0) + g[1] * v0 + g[1] * v0 + 1.0;
    const double nn = sf::root(n2);
    t.ok = t.ok && n2 > 0.0;
    t.b = sf::div(v0, nn);
    t.c = sf::rcp(nn);
    t.e2 = t.e3 = 1.0;
  } else {
    t.b = 0.0;
    t.c = g[5] == 1.0 ? 1.0 : sf::rcp(sf::root(g[5]));
    t.e2 = sf::rcp(sf::root(g[10]));
    t.e3 = sf::rcp(sf::root(g[15]));
    t.ok = t.ok && g[5] > 0.0 && g[10] > 0.0 && g[15] > 0.0;
  }
  return t;
}

// what: as curvature_kernel, 1 to 6. Blocks per SM: as many as the registers of the
// sparse path let in; the dense functions, which hardly a point calls, would set
// them for the whole kernel (156-166 registers and 6 blocks per SM: R at 60000 points
// 872 us for Alcubierre, 142 for Morris-Thorne, whole calls; 753 and 131 as it is).
template <int K, bool GRID>
__global__ void __launch_bounds__(POINT_THREADS, K == KIND_SCHWARZSCHILD ? 12 : 10)
curvature_point_kernel(const MetricDesc M, int what, const double* __restrict__ xs, int64_t n,
                       const double* __restrict__ ks, int64_t nk, int k_shared, double* __restrict__ out, int* flags,
                       const GridDesc grid, uint64_t seed, double* __restrict__ out2, double* __restrict__ kout) {
  using PM = PointMetric<K>;
  using ST = typename PM::ST;
  extern __shared__ double smem[];
  double* v = smem + threadIdx.x;                                // [NV][THREADS]
  double* diff = smem + PM::NV * POINT_THREADS + threadIdx.x;    // [axes][ND][THREADS]
  const int64_t pt = (int64_t)blockIdx.x * POINT_THREADS + threadIdx.x;
  if (pt >= n) return;  // no barrier below: every thread keeps to its own column
  double x[4];
  if (GRID) {
    grid_point(grid, pt, x);
  } else {
    x[0] = xs[4 * pt]; x[1] = xs[4 * pt + 1]; x[2] = xs[4 * pt + 2]; x[3] = xs[4 * pt + 3];
  }
  PM::values(M, x, v, diff);
  const double inv_2h = 1.0 / (2.0 * FD_H);
  double c[PM::NG];
  unsigned big = 0;
  bool regular = true;
  // slots from the last to the point itself, whose symbols stay in c; the minus
  // slot of an axis comes first and leaves its symbols in the store
#pragma unroll 1
  for (int sl = ST::slots - 1; sl >= 0; --sl) {
    regular &= PM::symbols(M, x, v, sl, c);
#pragma unroll
    for (int i = 0; i < PM::NG; ++i) {
      const unsigned h = 2u * sf::hi_of(c[i]);
      big = h > big ? h : big;
    }
    if (sl > 0) {
      double* row = diff + ((sl - 1) >> 1) * PM::ND * POINT_THREADS;
      const bool minus = ((sl - 1) & 1) != 0;
#pragma unroll
      for (int i = 0; i < PM::NG; ++i) {
        const int w = PM::diff_place(i);
        if (w >= 0) row[w * POINT_THREADS] = minus ? c[i] : (c[i] - row[w * POINT_THREADS]) * inv_2h;
      }
    }
  }
  double ric[16];
  const bool plain = regular && big < 2u * SYMBOL_BOUND;
  if (plain) {
    PM::ricci(c, [&](int axis, int i) { return diff[(axis * PM::ND + PM::diff_place(i)) * POINT_THREADS]; }, ric);
  } else {
    dense_ricci<K>(M, x, ric, flags);
  }
  if (what == 1) {
#pragma unroll
    for (int q = 0; q < 16; ++q) out[16 * pt + q] = ric[q];
    return;
  }
  double g[16] = {}, gi[16] = {};
  PM::metric(M, x, v, g, gi);
  if (!plain) {  // the dense inverse and its sums
    metric_g<K>(M, x, g);
    if (!metric_g_inv_given<K>(M, x, g, gi)) atomicOr(flags, 1);
  }
  double rs = 0.0;  // curvature.rs:87-97; g^-1 is zero where g is
#pragma unroll
  for (int q = 0; q < 16; ++q)
    if ((PM::GMASK >> q) & 1) rs += gi[q] * ric[q];
  if (!plain) {
    rs = 0.0;
    for (int q = 0; q < 16; ++q) rs += gi[q] * ric[q];
  }
  if (what == 2) {
    out[pt] = rs;
    return;
  }
  const double factor = 1.0 / (8.0 * 3.141592653589793);
  double ein[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) {  // curvature.rs:99-110
    ein[q] = ric[q];
    if ((PM::GMASK >> q) & 1) ein[q] = ric[q] - sf::half(g[q]) * rs;
    else if (!sf::finite(rs)) ein[q] = ric[q] - 0.0 * rs;
  }
  if (what == 3 || what == 4 || (what == 6 && out)) {
#pragma unroll
    for (int q = 0; q < 16; ++q) out[16 * pt + q] = what == 4 ? ein[q] * factor : ein[q];
    if (what <= 4) return;
  }
  double t[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) t[q] = ein[q] * factor;  // curvature.rs:112-122
  if (what == 6 && !plain) {
    dense_contractions(g, t, seed, pt, nk, out2, kout);
    return;
  }
  SparseTetrad tet = {};
  if (what == 6) tet = sparse_tetrad<K>(g);
  // T(k, k) (curvature.rs:127-136) of the point's vectors, one after another
#pragma unroll 1
  for (int64_t q = 0; q < nk; ++q) {
    double k[4];
    if (what == 6) {  // point_null_vector
      const uint64_t h = splitmix64(seed ^ (uint64_t)(pt * nk + q));
      const double u1 = sf::unit53(h >> 11), u2 = sf::unit53(splitmix64(h) >> 11);
      const double z = fma(2.0, u1, -1.0);  // 2 u1 is exact
      const double rho = sf::root(1.0 - z * z);  // not negative: |z| <= 1
      double sp, cp;
      dm::sincos_det(6.283185307179586 * u2, &sp, &cp);
      const double n1 = rho * cp, n2 = rho * sp;
      k[0] = K == KIND_ALCUBIERRE ? tet.a + n1 * tet.b : tet.a;
      k[1] = n1 * tet.c;
      k[2] = n2 * tet.e2;
      k[3] = z * tet.e3;
      if (!tet.ok) k[0] = k[1] = k[2] = k[3] = __longlong_as_double(0x7ff8000000000000LL);
      if (kout) {
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) kout[4 * (pt * nk + q) + mu] = k[mu];
      }
    } else {
      const double* kp = k_shared ? ks + 4 * q : ks + 4 * (pt * nk + q);
      k[0] = kp[0]; k[1] = kp[1]; k[2] = kp[2]; k[3] = kp[3];
    }
    double sacc = 0.0;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
#pragma unroll
      for (int nu = 0; nu < 4; ++nu) sacc += t[4 * mu + nu] * k[mu] * k[nu];
    (what == 6 ? out2 : out)[pt * nk + q] = sacc;
  }
}

template <int K>
constexpr bool has_point_kernel() {
  return K == KIND_ALCUBIERRE || K == KIND_MORRIS_THORNE || K == KIND_SCHWARZSCHILD;
}

template <int K, bool GRID>
static cudaError_t launch_point_k(const MetricDesc& M, int what, const double* x, int64_t n, const double* k,
                                  int64_t nk, int k_shared, double* out, int* flags, const GridDesc& grid,
                                  uint64_t seed, double* out2, double* kout, cudaStream_t s) {
  using PM = PointMetric<K>;
  constexpr int axes = PM::ST::k;
  const size_t smem = (size_t)(PM::NV + axes * PM::ND) * POINT_THREADS * sizeof(double);
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(curvature_point_kernel<K, GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr_set = true;
  }
  const int64_t blocks = (n + POINT_THREADS - 1) / POINT_THREADS;
  curvature_point_kernel<K, GRID><<<(unsigned)blocks, POINT_THREADS, smem, s>>>(M, what, x, n, k, nk, k_shared, out,
                                                                                flags, grid, seed, out2, kout);
  return cudaGetLastError();
}

template <int K, bool GRID>
static cudaError_t launch_curv_k(const MetricDesc& M, int what, const double* x, int64_t n, const double* k,
                                 int64_t nk, int k_shared, double* out, int* flags, const GridDesc& grid,
                                 uint64_t seed, double* out2, double* kout, cudaStream_t s) {
  if constexpr (has_point_kernel<K>()) {
    if (what != 0 && one_thread_per_point(K == KIND_ALCUBIERRE, GRID, n, what >= 5 ? nk : 0, device_sms()))
      return launch_point_k<K, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
  }
  const size_t smem = curv_smem_doubles<K>() * sizeof(double);
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(curvature_kernel<K, GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr_set = true;
  }
  const int64_t blocks = (n + CURV_PPB - 1) / CURV_PPB;
  curvature_kernel<K, GRID><<<(unsigned)blocks, CURV_THREADS, smem, s>>>(M, what, x, n, k, nk, k_shared, out,
                                                                         flags, grid, seed, out2, kout);
  return cudaGetLastError();
}

template <bool GRID>
static cudaError_t launch_curv(const MetricDesc& M, int what, const double* x, int64_t n, const double* k,
                               int64_t nk, int k_shared, double* out, int* flags, const GridDesc& grid,
                               uint64_t seed, double* out2, double* kout, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (M.kind) {
    case KIND_MINKOWSKI: return launch_curv_k<KIND_MINKOWSKI, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
    case KIND_SCHWARZSCHILD: return launch_curv_k<KIND_SCHWARZSCHILD, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
    case KIND_ALCUBIERRE: return launch_curv_k<KIND_ALCUBIERRE, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
    case KIND_MORRIS_THORNE: return launch_curv_k<KIND_MORRIS_THORNE, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
    case KIND_FIELD: return launch_curv_k<KIND_FIELD, GRID>(M, what, x, n, k, nk, k_shared, out, flags, grid, seed, out2, kout, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_curvature(const MetricDesc& M, int what, const double* x, int64_t n, const double* k,
                             int64_t nk, int k_shared, double* out, int* flags, cudaStream_t s) {
  GridDesc none;
  memset(&none, 0, sizeof none);
  return launch_curv<false>(M, what, x, n, k, nk, k_shared, out, flags, none, 0, nullptr, nullptr, s);
}

cudaError_t launch_curvature_grid(const MetricDesc& M, const GridDesc& grid, int64_t nk, uint64_t seed,
                                  double* einstein, double* nec, double* kout, int* flags, cudaStream_t s) {
  const int64_t n = grid.n[0] * grid.n[1] * grid.n[2];
  return launch_curv<true>(M, 6, nullptr, n, nullptr, nk, 0, einstein, flags, grid, seed, nec, kout, s);
}

}  // namespace geon

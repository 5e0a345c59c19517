// The mixed path's steppers with and without their fast steps (groups of planar
// steps under one combined test, groups of flat Alcubierre steps) on the same rays,
// compared after every group of steps, bit for bit.
#include "../geon_gb300/csrc/internal.h"
#define GEON_STEPPERS_ONLY
#include "../geon_gb300/csrc/trace_mixed.cu"

namespace geon {

template <class Stepper>
struct Separate : Stepper {
  static constexpr bool FAST = false;
};
template <class Stepper>
struct Counting : Stepper {
  int64_t fast = 0;
  __device__ __forceinline__ int fast_steps(const TraceLaunch& L, int left) {
    const int done = Stepper::fast_steps(L, left);
    fast += done;
    return done;
  }
};

// out[4 i]: 0 where the two agree throughout, else 1 + the steps at the end of the
// first group where they do not; then termination, steps, steps taken fast.
template <int K, int FEAT>
__global__ void __launch_bounds__(64) compare(const TraceLaunch L, int src, const double* y0, int64_t n, int64_t* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Counting<MixedStepper<K, FEAT>> a;
  Separate<MixedStepper<K, FEAT>> b;
  double y[8];
  for (int q = 0; q < 8; ++q) y[q] = y0[8 * i + q];
  a.rebind(L);
  b.rebind(L);
  a.set_source(src);
  b.set_source(src);
  a.load(L, y);
  b.load(L, y);
  if (src == SRC_ARRAY) {
    a.check_null(L, y);
    b.check_null(L, y);
  }
  int64_t na = 0, nb = 0, taken_a = 0, taken_b = 0, bad = 0;
  int ta = TERM_NONE, tb = TERM_NONE;
  while (ta == TERM_NONE && !bad) {  // at most max_steps / TRACE_INNER + 1 times: every group counts its steps
    na = group_steps(a, L, L.max_steps, na, ta, taken_a);
    nb = group_steps(b, L, L.max_steps, nb, tb, taken_b);
    uint32_t wa[16], wb[16];
    a.save(wa);
    b.save(wb);
    bool same = na == nb && ta == tb && taken_a == taken_b;
    for (int q = 0; q < 16; ++q) same &= wa[q] == wb[q] || ((FEAT & FEAT_NO_TIME) != 0 && q % 8 == 0);
    if (!same) bad = 1 + na;
  }
  out[4 * i] = bad;
  out[4 * i + 1] = ta;
  out[4 * i + 2] = taken_a;
  out[4 * i + 3] = a.fast;
}

}  // namespace geon

using namespace geon;

// config: 0 orbit plane, 1 the same without t (renders), 2 equatorial sweep, 3 and 4 the serving
// kernel's camera and equatorial rays, 5 no frame (Alcubierre)
extern "C" int compare_steps(geon_metric_t m, int config, const double* y0, long long n, double step,
                             long long max_steps, long long* out) {
  const TraceLaunch L = trace_launch_defaults(m, step, max_steps);
  double* dy = nullptr;
  int64_t* dout = nullptr;
  if (cudaMalloc(&dy, sizeof(double) * 8 * n) || cudaMalloc(&dout, sizeof(int64_t) * 4 * n)) return -1;
  cudaMemcpy(dy, y0, sizeof(double) * 8 * n, cudaMemcpyHostToDevice);
  const unsigned grid = (unsigned)((n + 63) / 64);
  constexpr int S = KIND_SCHWARZSCHILD, T = KIND_MORRIS_THORNE, A = KIND_ALCUBIERRE;
  constexpr int SERVE_S = FEAT_OWN | FEAT_PLANAR_DYN | FEAT_ORBIT_DYN | FEAT_DECIDE_DYN, SERVE = FEAT_OWN | FEAT_ORBIT_DYN;
  const int kind = L.M.kind;
  bool known = true;
  if (kind == S && config == 0) compare<S, FEAT_ORBIT><<<grid, 64>>>(L, SRC_ARRAY, dy, n, dout);
  else if (kind == S && config == 1) compare<S, FEAT_ORBIT | FEAT_NO_TIME><<<grid, 64>>>(L, SRC_ARRAY, dy, n, dout);
  else if (kind == S && config == 2) compare<S, FEAT_PLANAR><<<grid, 64>>>(L, SRC_EQUATORIAL, dy, n, dout);
  else if (kind == S && config == 3) compare<S, SERVE_S><<<grid, 64>>>(L, SRC_CAMERA, dy, n, dout);
  else if (kind == S && config == 4) compare<S, SERVE_S><<<grid, 64>>>(L, SRC_EQUATORIAL, dy, n, dout);
  else if (kind == T && config == 0) compare<T, FEAT_ORBIT><<<grid, 64>>>(L, SRC_ARRAY, dy, n, dout);
  else if (kind == T && config == 1) compare<T, FEAT_ORBIT | FEAT_NO_TIME><<<grid, 64>>>(L, SRC_ARRAY, dy, n, dout);
  else if (kind == T && config == 3) compare<T, SERVE><<<grid, 64>>>(L, SRC_CAMERA, dy, n, dout);
  else if (kind == A && config == 5) compare<A, 0><<<grid, 64>>>(L, SRC_ARRAY, dy, n, dout);
  else known = false;
  int rc = known ? (int)cudaDeviceSynchronize() : -2;
  if (rc == 0) rc = (int)cudaMemcpy(out, dout, sizeof(int64_t) * 4 * n, cudaMemcpyDeviceToHost);
  cudaFree(dy);
  cudaFree(dout);
  return rc;
}

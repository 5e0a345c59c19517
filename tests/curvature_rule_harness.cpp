// C entry point over curvature_rule.h for the CPU tests.
#include "curvature_rule.h"

extern "C" int point_kernel(int alcubierre, int grid, long long n, long long nk, int sms) {
  return geon::one_thread_per_point(alcubierre != 0, grid != 0, n, nk, sms);
}

// Which curvature kernel a batch of points runs: one thread per point, or 16
// points per block of 128 threads. Host code (the CPU tests compile it with g++).
#pragma once
#include <cstdint>

namespace geon {

// Whether one thread per point is the faster kernel for n points with nk vectors
// each (Alcubierre; or Morris-Thorne and Schwarzschild). Its time is one thread's
// chain of operations until the points fill the SMs, the block kernel's goes by
// waves of blocks (96 points per SM for a grid, 128 for points of the caller's).
// us, one thread per point / block kernel, 152 SMs:
//  - Alcubierre, a box with the bubble's wall in it (warps with points on both
//    sides of a branch of tanh take both): grids of 9261 points 223 / 178, 13824
//    237 / 191, 19683 234 / 282; scattered points 9728 270 / 168, 19456 291 / 229,
//    24320 306 / 292, 38912 371 / 420 (whole calls). So from the second wave on.
//  - Morris-Thorne (Schwarzschild alike): 5120 points 34 / 79, 9728 37 / 97, 19456
//    36 / 187; the chain is short and there is no branch.
//  - Vectors: one thread takes a point's vectors one after another (3.7 us a vector
//    up to 64 points per SM, 4.2 up to 128), the block kernel spreads them over its
//    threads (0.26 ns a point and vector): Morris-Thorne 5120 points with 16 / 64 / 256
//    vectors 93 / 109, 270 / 200, 982 / 568; 9728 with 64 / 256 271 / 261, 981 / 753;
//    14592 with 256 / 1024 1120 / 1124, 4371 / 4078; 19456 with 256 1120 / 1497. The
//    crossing lies at nk (112 - points per SM) = 2100, and for Alcubierre grids at
//    1100 (14592 points: nk = 87).
inline bool one_thread_per_point(bool alcubierre, bool grid, int64_t n, int64_t nk, int sms) {
  const int64_t least = alcubierre ? (grid ? (int64_t)96 * sms + 1 : (int64_t)128 * sms + 1) : (int64_t)33 * sms;
  if (n < least) return false;
  const int64_t free = (int64_t)112 * sms - n;
  if (free <= 0 || nk <= 0) return true;
  return nk <= (alcubierre ? 1100 : 2100) * (int64_t)sms / free;
}

}  // namespace geon

// Which kernel a mixed shadow sweep runs: the launch variant a caller or the
// autotuner chose, or the rule on the number of rays. Host code (the CPU tests
// compile it with g++).
#pragma once
#include <cstdint>

namespace geon {

// Launch variants 0 to 8 of the equatorial shadow kernel are a register cap (none,
// 64, 51 registers) + 3 x block size (128, 64, 256 threads), at every number of
// rays; SWEEP_BY_SIZE, the default, leaves the choice to sweep_kernel.
constexpr int SWEEP_VARIANTS = 9;
constexpr int SWEEP_BY_SIZE = 9;
// Kernels that only the rule chooses: constants in registers and separate tests
// (FEAT_CHAIN), and one-warp blocks dealt by SM quarter (trace_resident).
constexpr int SWEEP_CHAIN = 10;
constexpr int SWEEP_RESIDENT = 11;

// A variant and the number of rays above which it holds (at and below: by size),
// in one word so that it is read and written at once.
inline int64_t sweep_choice(int variant, int64_t above) { return (int64_t)variant | (above < 0 ? 0 : above) << 4; }
inline int sweep_choice_variant(int64_t choice) { return (int)(choice & 15); }
inline int sweep_variant(int64_t choice, int64_t n) {
  return n > (choice >> 4) ? sweep_choice_variant(choice) : SWEEP_BY_SIZE;
}

// Rays that give every SM quarter one warp, and the most the GPU holds at once.
inline int64_t sweep_one_warp(int sms) { return (int64_t)sms * 128; }
inline int64_t sweep_held(int sms) { return (int64_t)sms * 1024; }

// Claimed longest first? Up to two warps per SM quarter (256 rays per SM) a sweep
// takes as long as its longest rays either way (20000 to 38900 rays 19.8 ms); from
// the third warp on the order keeps the long rays apart (41000 / 60000 / 120000 rays
// 20.0 / 20.3 / 36.8 ms in order, 27.6 / 36.0 / 60.6 not; 2^20 rays 269 and 290). The
// order's indexes are 32-bit.
inline bool sweep_ordered(int64_t n, int sms) { return n > 2 * sweep_one_warp(sms) && n < ((int64_t)1 << 31); }

// The kernel of a sweep of n rays. `resident`: the launch has trace_resident's
// workspace.
//  - One warp per SM quarter: the chain of a step sets the time (19000 rays 17.0
//    against 17.3 ms; from two warps on the combined test is the faster one:
//    38000 rays 21.9 against 22.9 ms).
//  - Everything held at once (32 one-warp blocks per SM): dealt by quarter (60000 /
//    120000 rays 20.3 / 36.8 ms; 28.9 / 46.2 from the queue, both longest first).
//  - More rays: the queue, with blocks of 64 threads, or of 128 at 51 registers and
//    a tenth block per SM once the rays are over twice the lanes (300000 rays 80.7
//    against 88.6 ms, 2^20 rays 270.2 against 267.3).
inline int sweep_kernel(int variant, int64_t n, int sms, bool resident) {
  if (variant != SWEEP_BY_SIZE) return variant;
  if (n <= sweep_one_warp(sms)) return SWEEP_CHAIN;
  if (resident) return SWEEP_RESIDENT;
  return n > 18 * sweep_one_warp(sms) ? 2 : 3;
}

// The autotuner's choice from the rates of the nine variants at n rays: by size
// unless a variant beats the queue kernel that the rule runs there by more than
// timing noise. At sizes the GPU holds at once the rule's kernels are none of the
// nine, so nothing is chosen; a choice holds where the queue runs.
inline int64_t sweep_tuned(const double* rates, int64_t n, int sms) {
  if (n <= sweep_held(sms)) return sweep_choice(SWEEP_BY_SIZE, 0);
  int best = sweep_kernel(SWEEP_BY_SIZE, n, sms, false);
  const double need = 1.02 * rates[best];
  bool better = false;
  for (int v = 0; v < SWEEP_VARIANTS; ++v)
    if (rates[v] > need && (!better || rates[v] > rates[best])) best = v, better = true;
  return better ? sweep_choice(best, sweep_held(sms)) : sweep_choice(SWEEP_BY_SIZE, 0);
}

}  // namespace geon

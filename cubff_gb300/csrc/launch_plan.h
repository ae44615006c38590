// launch_plan.h — how a pipelined launch is laid out on the device.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "common.cuh"
#include "internal.h"

namespace cubff {

// How many pairs a warp of a pipelined launch holds, and the warps per SM that such
// a launch has to keep busy to be chosen before narrower ones (0: all that are
// resident).
struct PipeWidth {
  uint32_t pairs, warps_per_sm;
};

// The widths of a language's kernels.  A wide warp runs the first stages of its
// pairs for the price of a narrow one's, but its long pairs wait for one another;
// so a launch is wide when there are pairs enough to keep as many warps busy.
//  * The BFF languages with matched brackets run every long pair on a whole warp:
//    all resident warps (16 soups of 2^13 to 2^17 bff programs, 128 epochs from a
//    random start: 57 ms; 8 pairs to a warp 87, one pair a lane 80).
//  * Where the lanes of a warp may take long pairs on side by side, 3 warps to an SM
//    are enough: Forth (64 epochs of 2^17 forth programs: 18 ms, 8 pairs to a warp
//    22; of 2^15 it is the other way round, 10.6 and 9.8) and, 16 to a warp, bff8
//    (2^17 programs evolved for 4096 epochs: 136 ms, 178), which takes 32 only when
//    all resident warps have them.
//  * SUBLEQ: 16 (LaneServer).
constexpr int kPipeWidths = 3;
struct PipeWidths {
  int count;
  PipeWidth width[kPipeWidths];
};
constexpr PipeWidths pipe_widths(int lang) {
  if (lang == kBff8 || lang == kBff8Noheads) return {3, {{8, 0}, {16, 3}, {32, 0}}};
  if (lang <= kBffSelfmove) return {2, {{8, 0}, {32, 0}}};
  if (lang <= kForthtrivialReset) return {2, {{8, 0}, {32, 3}}};
  return {1, {{16, 0}}};
}

// One pipelined kernel.
struct PipeKernel {
  const void *fn;
  size_t smem;  // shared memory of a block, but for the soups' descriptors
  size_t smem_bytes(int n_soups) const { return smem + size_t(n_soups) * sizeof(PipeSoup); }
};
// A language's kernels, by width.
struct PipeKernels {
  PipeKernel kernel[kPipeWidths];
};

struct PipePlan {
  int which;      // of the language's widths
  uint32_t grid;  // blocks of kPipeWarps warps
};
constexpr uint32_t kPipeWarps = 4;

// Whether a busy warp claims new pairs when so many of the `width` lanes that hold
// pairs are idle: claim_min of 32, in proportion.
__host__ __device__ constexpr bool idle_enough(uint32_t idle, uint32_t width, uint32_t claim_min) {
  return idle * 32 >= claim_min * width;
}

// Lanes in flight: enough to keep the SMs busy, few enough that most held
// pairs are ready (a lane holding a pair of a later epoch only polls).
// lanes_per_pair64 (x1/64) is tunable; the default, kDefaultLanes, keeps half an
// epoch of pairs in flight.  With that or more of them a launch has at least
// kMinLanesPerSm to an SM, if it has as many pairs: so few warps disturb each other
// little, so of a small soup all pairs of an epoch are in flight (64 epochs of 1022
// bff_noheads programs: 1.74 ms, with half of them 2.05; of 8192: 2.49, 2.62; of
// 16384, where it would be twice as many warps: 3.61, 3.49).  A caller who asks for
// fewer, to leave room for other work, gets them.
constexpr uint32_t kDefaultLanes = 32, kMinLanesPerSm = 27;
inline uint64_t lanes_wanted(uint64_t total_pairs, uint32_t lanes_per_pair64, int sms) {
  const uint64_t per64 = lanes_per_pair64 ? lanes_per_pair64 : kDefaultLanes;
  const uint64_t want = std::max<uint64_t>(1, total_pairs * per64 / 64);
  if (per64 < kDefaultLanes) return want;
  return std::max<uint64_t>(want, std::min<uint64_t>(total_pairs, uint64_t(kMinLanesPerSm) * sms));
}

// Which width a launch of so many lanes takes.
inline int choose_width(const PipeWidths &w, uint64_t lanes, int sms, int narrow_per_sm) {
  const uint64_t resident = uint64_t(kPipeWarps) * std::max(1, narrow_per_sm);
  int which = 0;
  for (int i = 1; i < w.count; i++)
    if (lanes >= sms * (w.width[i].warps_per_sm ? w.width[i].warps_per_sm : resident) * w.width[i].pairs)
      which = i;
  return which;
}

// The blocks of it, of which per_sm are resident on an SM.
inline uint32_t grid_of(const PipeWidth &w, uint64_t lanes, int sms, int per_sm) {
  const uint64_t per_block = uint64_t(kPipeWarps) * w.pairs;
  const uint64_t resident = uint64_t(sms) * std::max(1, per_sm);
  return static_cast<uint32_t>(std::min((lanes + per_block - 1) / per_block, resident));
}

}  // namespace cubff

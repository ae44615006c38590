// Test harness: how a pipelined launch is laid out (launch_plan.h), on the host.
#include "launch_plan.h"

using namespace cubff;

extern "C" int claims(uint32_t idle, uint32_t width, uint32_t claim_min) {
  return idle_enough(idle, width, claim_min);
}

// Pairs to a warp and blocks of a launch of total_pairs pairs, with narrow_per_sm
// blocks of the narrow kernel and per_sm of the chosen one resident on an SM.
extern "C" void launch_plan(int lang, uint64_t total_pairs, uint32_t lanes_per_pair64, int sms,
                            int narrow_per_sm, int per_sm, uint32_t *pairs, uint32_t *grid) {
  const PipeWidths w = pipe_widths(lang);
  const uint64_t lanes = lanes_wanted(total_pairs, lanes_per_pair64, sms);
  const int which = choose_width(w, lanes, sms, narrow_per_sm);
  *pairs = w.width[which].pairs;
  *grid = grid_of(w.width[which], lanes, sms, which ? per_sm : narrow_per_sm);
}

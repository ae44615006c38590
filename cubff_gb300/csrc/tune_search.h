// tune_search.h — the launch-shape tuner's search, apart from what it times.
#pragma once

#include <cstdint>

#include "cubff_gb300.h"

namespace cubff {

// Two runs of one launch differ by a few percent; a shape has to be faster than the
// best so far by more to take its place.
constexpr double kTuneMargin = 0.97;

// Coordinate descent from *best: each knob in turn over a short list of values, the
// others fixed; two passes.  Launches whose lanes run steps by visits (SUBLEQ) have
// all five knobs, the others the lanes in flight alone.  time_of(shape, &seconds)
// times a shape (nonzero: stop); same(a, b) tells that two shapes give the same
// launch, so that the second need not be timed.
template <class TimeOf, class Same>
int search_shape(bool visits, cubff_tuning *best, TimeOf time_of, Same same) {
  static const uint32_t kValues[5][5] = {{16, 24, 32, 48, 64},     // lanes_per_pair64
                                         {16, 32, 64, 128, 256},   // steps_per_visit
                                         {8, 14, 20, 26, 32},      // claim_min
                                         {0, 1, 2, 4, 8},          // long_visits
                                         {4, 8, 16, 32, 64}};      // first_visit_steps
  uint32_t cubff_tuning::*const kKnobs[5] = {
      &cubff_tuning::lanes_per_pair64, &cubff_tuning::steps_per_visit, &cubff_tuning::claim_min,
      &cubff_tuning::long_visits, &cubff_tuning::first_visit_steps};
  const int knobs = visits ? 5 : 1, passes = visits ? 2 : 1;
  double best_s = 0;
  if (const int st = time_of(*best, &best_s)) return st;
  for (int pass = 0; pass < passes; pass++) {
    for (int knob = 0; knob < knobs; knob++) {
      const cubff_tuning base = *best;
      double limit = best_s * kTuneMargin;
      for (const uint32_t v : kValues[knob]) {
        cubff_tuning cand = base;
        cand.*kKnobs[knob] = v;
        if (same(cand, base) || (knob == 0 && same(cand, *best))) continue;
        double sec = 0;
        if (const int st = time_of(cand, &sec)) return st;
        if (sec < limit) {
          limit = best_s = sec;
          *best = cand;
        }
      }
    }
  }
  return 0;
}

}  // namespace cubff

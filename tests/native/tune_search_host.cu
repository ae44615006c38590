// Test harness: the tuner's search (tune_search.h) over made-up times.
#include "tune_search.h"

using namespace cubff;

// Searches from *shape with the callback's times; launches whose lanes_per_pair64 are
// both at least lanes_same are the same.  Returns the number of shapes timed.
extern "C" int tune_search(int visits, cubff_tuning *shape, double (*time_of)(const cubff_tuning *),
                           uint32_t lanes_same) {
  int timed = 0;
  search_shape(
      visits != 0, shape,
      [&](const cubff_tuning &t, double *s) {
        timed++;
        *s = time_of(&t);
        return 0;
      },
      [&](const cubff_tuning &a, const cubff_tuning &b) {
        const bool lanes = a.lanes_per_pair64 == b.lanes_per_pair64 ||
                           (a.lanes_per_pair64 >= lanes_same && b.lanes_per_pair64 >= lanes_same);
        return lanes && (!visits || (a.steps_per_visit == b.steps_per_visit &&
                                     a.claim_min == b.claim_min && a.long_visits == b.long_visits &&
                                     a.first_visit_steps == b.first_visit_steps));
      });
  return timed;
}

// Test harness: the engine's mutation draws (common.cuh), compiled for the host.
#include "common.cuh"

// Draws from each of n keys; returns how many words differ from draws one by one.
extern "C" uint64_t mutation_words_differ(const uint64_t *keys, uint64_t n, uint32_t prob) {
  uint64_t bad = 0;
  for (uint64_t i = 0; i < n; i++) {
    uint32_t want = 0;
    for (int b = 0; b < 32; b++) {
      const uint64_t r = cubff::splitmix64(keys[i] + b);
      want |= static_cast<uint32_t>(((r >> 8) & ((1ull << 30) - 1)) < prob) << b;
    }
    bad += cubff::mutation_word(keys[i], prob) != want;
  }
  return bad;
}

// common.cuh — shared device/host definitions of the cubff GB300 engine.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace cubff {

constexpr int kTape = 64;             // kSingleTapeSize (common.h:55)
constexpr int kPair = 2 * kTape;      // one pair tape
constexpr int kStepLimit = 8 * 1024;  // Evaluate(tape, 8 * 1024) (common_language.h:184)
constexpr int kNumLangs = 13;

// Language ids, in the order of the reference's registered names.
enum Lang : int {
  kBff = 0,
  kBffNoheads,
  kBffNoheads4bit,
  kBffPerm,
  kBff8,
  kBff8Noheads,
  kBffSelfmove,
  kForth,
  kForthcopy,
  kForthtrivial,
  kForthtrivialReset,
  kSubleq,
  kRsubleq4,
};

// SplitMix64 finaliser (Steele, Lea, Flood, OOPSLA 2014), the RNG of
// common_language.h:131-136.
__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  uint64_t z = x + 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

// seed(x) = SplitMix64(SplitMix64(params.seed) ^ SplitMix64(x))
// (common_language.h:367-369); s0 = SplitMix64(params.seed).
__host__ __device__ __forceinline__ uint64_t seed_from(uint64_t s0, uint64_t x) {
  return splitmix64(s0 ^ splitmix64(x));
}

// The 32 draws from key0 on of a pair's mutations (common_language.h:172-180) as
// a word: bit b is set iff bits [8, 38) of SplitMix64(key0 + b) are below prob,
// and byte b of the 32 becomes the draw's low byte.  What the keys have in common
// is taken out: the high half of the sum, its share of the first product, and the
// shifted-in bits; so a draw is some 16 instructions instead of 25.  (The masks of
// 20 epochs of 2^17 programs: 129 us, 171 draw by draw.)
__host__ __device__ __forceinline__ uint32_t mutation_word(uint64_t key0, uint32_t prob) {
  if (prob >= 1u << 30) return ~0u;
  const uint64_t z0 = key0 + 0x9e3779b97f4a7c15ULL;
  const uint32_t lo = static_cast<uint32_t>(z0), hi = static_cast<uint32_t>(z0 >> 32);
  uint32_t m = 0;
  if ((lo >> 30) != ((lo + 31) >> 30)) {  // the keys differ above bit 29
    for (int b = 0; b < 32; b++)
      m |= static_cast<uint32_t>(
               (static_cast<uint32_t>(splitmix64(key0 + b) >> 8) & ((1u << 30) - 1)) < prob) << b;
    return m;
  }
  const uint32_t in = hi << 2 | lo >> 30;  // the low half of z >> 30
  const uint64_t of_hi = static_cast<uint64_t>((hi ^ (hi >> 30)) * 0x1ce4e5b9u) << 32;
#pragma unroll 8
  for (int b = 0; b < 32; b++) {
    const uint32_t x = (lo + b) ^ in;
    uint64_t z = static_cast<uint64_t>(x) * 0x1ce4e5b9u + of_hi;
    z += static_cast<uint64_t>(x * 0xbf58476du) << 32;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    // Bits [6, 38) of the draw: prob * 4 has none of the lowest two.
    const uint32_t v = static_cast<uint32_t>(z >> 6) ^ static_cast<uint32_t>(z >> 37);
    m |= static_cast<uint32_t>(v < prob * 4) << b;
  }
  return m;
}

// Shared-memory tape layout.  Threads come in groups of four warps.  The
// four warps of a group share one 16 KiB block in which byte p of the tape of
// lane l of warp w sits at  p * 128 + l * 4 + (w & 3):  every lane of a warp
// always hits its own bank (bank = l), whatever positions the 32 lanes touch,
// and the byte offset of position p is one shift-add from the thread's base.
constexpr int kGroupBytes = kPair * 128;  // 16 KiB per four warps

__device__ __forceinline__ uint32_t lane_base(uint32_t tid) {
  const uint32_t warp = tid >> 5, lane = tid & 31;
  return (warp >> 2) * kGroupBytes + lane * 4 + (warp & 3);
}

// One thread's 128-byte tape (or 128-byte stack) in the layout above.
// Positions are taken mod 128 (one AND), so no index a caller computes can
// leave the thread's own 128 bytes: every interpreter keeps its positions in
// 0..127 anyway, and the parity tests would show any position that relied on
// the wrap.
#ifdef CUBFF_HOST_INDEX_CHECK
// Host-compiled analysis builds only: reports every position outside the
// accessor's range before it is wrapped or clamped.
void cubff_index_violation(int kind, int p);
#define CUBFF_CHECK_POS(kind, p, hi) \
  do { if ((p) < 0 || (p) > (hi)) cubff_index_violation((kind), (p)); } while (0)
#else
#define CUBFF_CHECK_POS(kind, p, hi) do { } while (0)
#endif

struct LaneBytes {
  uint8_t *s;     // dynamic shared memory block holding the layout
  uint32_t base;  // lane_base(tid)
  __host__ __device__ __forceinline__ uint32_t get(int p) const {
    CUBFF_CHECK_POS(0, p, kPair - 1);
    return s[base + ((static_cast<uint32_t>(p) & (kPair - 1)) << 7)];
  }
  __host__ __device__ __forceinline__ void set(int p, uint32_t v) const {
    CUBFF_CHECK_POS(1, p, kPair - 1);
    s[base + ((static_cast<uint32_t>(p) & (kPair - 1)) << 7)] = static_cast<uint8_t>(v);
  }
};

// The tapes of `stride` lanes of a warp as interleaved words: byte p of lane l
// sits at (p / 4 * stride + l) * 4 + p % 4 of a block of stride * 128 bytes, so a
// tape is staged and written back a word at a time.
template <uint32_t stride>
struct LaneWords {
  uint8_t *s;     // the block, 4-byte aligned
  uint32_t lane;
  __host__ __device__ __forceinline__ uint32_t get(int p) const { return s[at(p)]; }
  __host__ __device__ __forceinline__ void set(int p, uint32_t v) const {
    s[at(p)] = static_cast<uint8_t>(v);
  }
  __host__ __device__ __forceinline__ uint32_t at(int p) const {
    const uint32_t x = static_cast<uint32_t>(p) & (kPair - 1);
    return ((x >> 2) * stride + lane) * 4 + (x & 3);
  }
  __host__ __device__ __forceinline__ uint32_t &word(uint32_t w) const {
    return reinterpret_cast<uint32_t *>(s)[w * stride + lane];
  }
};

// A per-thread array that the interpreters' common interface passes along
// (kNpBytes per 128 threads); none uses it any more.
constexpr int kNpEntries = kPair + 1;
constexpr int kNpBytes = kNpEntries * 128 * 2;
struct LaneNp {
  uint16_t *s;
  uint32_t base;
};

}  // namespace cubff

// subleq.cuh — SUBLEQ (subleq.cu:109-133) and RSUBLEQ4 (rsubleq4.cu:116-141)
// as resumable machines, with exact cycle fast-forward: at every step whose next
// position is not past the current one the state (pos, tape) is compared with a
// Brent-schedule snapshot.  The snapshot is a copy of the tape, and each write
// keeps the number of positions that differ from it, so that a comparison is one
// of counters.
//
// A step is a chain of two dependent loads (code, then operands) and the
// arithmetic between them, without a branch but for the rare visit(); a lone long
// program takes 190 cycles a step.  (With a mask of the positions written since
// the snapshot, a byte-wise comparison of those and a load per code byte: 455,
// RSUBLEQ4 312.)
#pragma once

#include "cycle.cuh"

namespace cubff {

// Backward steps before the first snapshot: few random programs take as many.
constexpr uint32_t kFirstSnapshot = 8;

// The n bytes from pos on, the first in the low byte: of a tape in words by two
// loads (what lies past the n bytes is any).
template <int n>
__host__ __device__ __forceinline__ uint32_t code_at(const LaneBytes t, int pos) {
  uint32_t c = 0;
#pragma unroll
  for (int q = 0; q < n; q++) c |= t.get(pos + q) << (8 * q);
  return c;
}
template <int n, uint32_t stride>
__host__ __device__ __forceinline__ uint32_t code_at(const LaneWords<stride> t, int pos) {
  const uint32_t w = static_cast<uint32_t>(pos) >> 2;
  const uint32_t lo = t.word(w), hi = t.word((w + 1) % (kPair / 4));
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, pos * 8);  // (by pos * 8 mod 32)
#else
  return static_cast<uint32_t>((static_cast<uint64_t>(hi) << 32 | lo) >> ((pos & 3) * 8));
#endif
}

// Copies tape t to s.
__host__ __device__ __forceinline__ void copy_tape(const LaneBytes t, const LaneBytes s) {
  for (int p = 0; p < kPair; p++) s.set(p, t.get(p));
}
template <uint32_t stride>
__host__ __device__ __forceinline__ void copy_tape(const LaneWords<stride> t,
                                                   const LaneWords<stride> s) {
#pragma unroll 8
  for (uint32_t w = 0; w < kPair / 4; w++) s.word(w) = t.word(w);
}

// B: a tape's bytes, LaneBytes or LaneWords.
template <bool kRelative4>
struct SubleqMachine {
  int pos;
  uint32_t i, mods;
  int s_pos;      // of the snapshot; kPair: there is none yet
  uint32_t s_i;
  int diff;       // positions whose byte is not the snapshot's
  uint32_t left;  // backward steps until the next snapshot
  uint32_t power;

  __host__ __device__ __forceinline__ void begin() {
    pos = 0;
    i = mods = 0;
    s_pos = kPair;
    s_i = 0;
    diff = 0;
    left = power = kFirstSnapshot;
  }

  // One step; returns true when the program has ended (every step counts).  The
  // jump's target counts as written by this step, but is loaded before the write,
  // with the operands.
  template <class B>
  __host__ __device__ __forceinline__ bool step(const B t, const B snap) {
    constexpr int kLen = kRelative4 ? 4 : 3;
    const int prev = pos;
    const uint32_t code = code_at<kLen>(t, pos);
    const int from = kRelative4 ? prev : 0;
    const int a = (from + code) & (kPair - 1);
    const int b = (from + (code >> 8)) & (kPair - 1);
    const uint32_t o = t.get(a), was = snap.get(a);
    const uint32_t v =
        (kRelative4 ? t.get(b) - t.get((from + (code >> 16)) & (kPair - 1)) : o - t.get(b)) & 0xFF;
    t.set(a, v);
    mods |= v ^ o;
    diff += (v != was) - (o != was);
    const uint32_t target = a == prev + kLen - 1 ? v : (code >> (8 * kLen - 8)) & 0xFF;
    const int to = kRelative4 ? prev + static_cast<int8_t>(target) : static_cast<int>(target);
    pos = static_cast<int8_t>(v) <= 0 ? to : prev + kLen;
    i++;
    const bool back = pos <= prev;
    left -= back;
    if (back && (left == 0 || (pos == s_pos && diff == 0))) visit(t, snap);
    return pos + kLen > kPair || pos < 0 || i >= kStepLimit;
  }

  // A backward step that finds the snapshot's state or is due to renew it.
  template <class B>
  __host__ __device__ __forceinline__ void visit(const B t, const B snap) {
    if (pos == s_pos && diff == 0) i += (kStepLimit - i) / (i - s_i) * (i - s_i);
    if (left != 0) return;
    copy_tape(t, snap);
    s_pos = pos;
    s_i = i;
    diff = 0;
    power *= 2;
    left = power;
  }

  __host__ __device__ __forceinline__ uint32_t ops() const { return i; }
  __host__ __device__ __forceinline__ uint32_t raw() const { return i; }
};

__host__ __device__ __forceinline__ uint32_t subleq_eval(const LaneBytes t, const LaneBytes snapa,
                                                         uint32_t *raw) {
  SubleqMachine<false> m;
  m.begin();
  while (!m.step(t, snapa)) {
  }
  *raw = m.raw();
  return m.ops();
}

__host__ __device__ __forceinline__ uint32_t rsubleq4_eval(const LaneBytes t, const LaneBytes snapa,
                                                           uint32_t *raw) {
  SubleqMachine<true> m;
  m.begin();
  while (!m.step(t, snapa)) {
  }
  *raw = m.raw();
  return m.ops();
}

}  // namespace cubff

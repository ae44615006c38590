// interp.cuh — compile-time dispatch to the 13 language interpreters.
// Every interpreter runs Language::Evaluate(tape, 8192) and gives the
// reference-counted op count (Evaluate's return value) and the raw loop
// iterations.
#pragma once

#include <type_traits>

#include "bff.cuh"
#include "forth.cuh"
#include "languages.cuh"
#include "subleq.cuh"

namespace cubff {

template <int L>
struct LangTraits {
  static constexpr bool kStaged = (L <= kForthtrivialReset);  // BFF and Forth families
};

// The two machines that run a BFF or Forth program in turn: on a lane, then on
// a warp (with that warp's shared memory, and whether a program has a stack).
template <int L, bool kBff = (L <= kBffSelfmove)>
struct Stages {
  static constexpr int kLogic = (L == kBff8 || L == kBff8Noheads)
                                    ? kLogicJump8
                                    : (L == kBffSelfmove ? kLogicSelfmove : kLogicScan);
  static constexpr uint32_t kNullMask = L == kBffNoheads4bit ? 0x0Fu : 0xFFu;
  using Lane = BffLane<(L == cubff::kBff || L == kBffPerm || L == kBff8 || L == kBffSelfmove),
                       kLogic, kNullMask>;
  template <class W>
  using Warp = BffWarp<W, kLogic, kNullMask>;
  using Mem = BffMem;
  using State = BffState;
  static constexpr bool kStack = false;
  // Whether the lanes of a warp may take on their long pairs side by side (not where
  // the warp runs loops by many iterations at a time), and how many of its pairs
  // have to go on past their first stage for that.
  static constexpr bool kCrowds = kLogic == kLogicJump8;
  __host__ __device__ static constexpr int crowd(int pairs) { return pairs == 8 ? 8 : pairs * 7 / 8; }
  // The last so many of them run on the whole warp all the same, which is several
  // times as fast for one alone.
  __host__ __device__ static constexpr int last(int pairs) { return pairs / 8; }
};
template <int L>
struct Stages<L, false> {
  using Lane = ForthFirst<(L == kForthtrivialReset)>;
  template <class W>
  using Warp = ForthWarp<W, (L == kForthtrivialReset)>;
  using Mem = ForthMem;
  using State = ForthState;
  static constexpr bool kStack = true;
  static constexpr bool kCrowds = true;
  __host__ __device__ static constexpr int crowd(int pairs) { return pairs * 6 / 8; }
  __host__ __device__ static constexpr int last(int) { return 0; }  // (no faster there)
};

// A resumable SUBLEQ interpreter of language L behind one interface: begin()
// on a staged tape, step() until it returns true, then ops() / raw().
template <int L, bool kStaged = (L <= kForthtrivialReset)>
struct LaneMachine {
  SubleqMachine<(L == kRsubleq4)> m;

  __host__ __device__ __forceinline__ void begin(const LaneBytes, Mask128) { m.begin(); }
  __host__ __device__ __forceinline__ bool step(const LaneBytes t, const LaneBytes stk,
                                                const LaneNp, const uint8_t *) {
    return m.step(t, stk);
  }
  __host__ __device__ __forceinline__ uint32_t ops() const { return m.ops(); }
  __host__ __device__ __forceinline__ uint32_t raw() const { return m.raw(); }
  __host__ __device__ __forceinline__ uint32_t mods() const { return m.mods; }
};

// The same interface over the two stages, on the host: a step of the lane's, or
// all of the warp's.
template <int L>
struct LaneMachine<L, true> {
  using Lane = typename Stages<L>::Lane;
  Lane lane;
  Mask128 cmd;
  bool begun;
  uint32_t n, i;

  void begin(const LaneBytes, Mask128 cmd_mask) {
    cmd = cmd_mask;
    begun = false;
    n = i = 0;
  }
  bool step(const LaneBytes t, const LaneBytes stk, const LaneNp, const uint8_t *optab) {
    if (!begun) lane.begin(t, cmd, optab);
    else lane.step(t, stk, optab);
    begun = true;
    if (lane.status == Lane::kJumps) lane.resolve(t, optab);
    n = lane.ops();
    i = lane.raw();
    if (lane.status == Lane::kJumps) {
      typename Stages<L>::Mem mem;
      for (int p = 0; p < kPair; p++) {
        mem.T[p] = static_cast<uint8_t>(t.get(p));
        if constexpr (Stages<L>::kStack) mem.stk[p] = static_cast<uint8_t>(stk.get(p));
      }
      typename Stages<L>::template Warp<HostWarp> warp(HostWarp{}, mem, optab);
      warp.run(lane.state());
      for (int p = 0; p < kPair; p++) t.set(p, mem.T[p]);
      n = warp.ops();
      i = warp.raw();
      return true;
    }
    return lane.status == Lane::kEnds;
  }
  uint32_t ops() const { return n; }
  uint32_t raw() const { return i; }
};

// Language::Evaluate on one tape: on a thread (SUBLEQ), or on the host.
template <int L>
__host__ __device__ __forceinline__ uint32_t evaluate(const LaneBytes t, const LaneBytes stk,
                                                      const uint8_t *__restrict__ optab,
                                                      uint32_t *raw) {
  if constexpr (L == kSubleq) {
    return subleq_eval(t, stk, raw);
  } else if constexpr (L == kRsubleq4) {
    return rsubleq4_eval(t, stk, raw);
  } else {
    LaneMachine<L> m;
    Mask128 cmd{0, 0};
    for (int p = 0; p < kPair; p++) mask_assign(cmd, p, op_of(L, t.get(p)) < kNull);
    m.begin(t, cmd);
    while (!m.step(t, stk, LaneNp{nullptr, 0}, optab)) {
    }
    *raw = m.raw();
    return m.ops();
  }
}

}  // namespace cubff

// interp.cuh — compile-time dispatch to the 13 language interpreters.
// Every interpreter runs Language::Evaluate(tape, 8192) on one thread's
// shared-memory pair tape and returns the reference-counted op count
// (Evaluate's return value), reporting the raw loop iterations in *raw.
#pragma once

#include <type_traits>

#include "bff.cuh"
#include "forth.cuh"
#include "languages.cuh"
#include "subleq.cuh"

namespace cubff {

// ---------------------------------------------------------------------------
// Per-language dispatch (compile-time).

template <int L>
struct LangTraits {
  static constexpr bool kForthFamily = (L >= kForth && L <= kForthtrivialReset);
  static constexpr bool kNeedsTable = (L <= kForthtrivialReset);
};

template <int L>
__host__ __device__ __forceinline__ uint32_t evaluate(const LaneBytes t, const LaneBytes stk,
                                             const uint8_t *__restrict__ optab,
                                             uint32_t *raw) {
  if constexpr (L == kBff) return bff_eval<true, kLogicScan, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kBffNoheads) return bff_eval<false, kLogicScan, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kBffNoheads4bit) return bff_eval<false, kLogicScan, 0x0F>(t, stk, optab, raw);
  else if constexpr (L == kBffPerm) return bff_eval<true, kLogicScan, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kBff8) return bff_eval<true, kLogicJump8, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kBff8Noheads) return bff_eval<false, kLogicJump8, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kBffSelfmove) return bff_eval<true, kLogicSelfmove, 0xFF>(t, stk, optab, raw);
  else if constexpr (L == kForthtrivialReset) return forth_eval<true>(t, stk, optab, raw);
  else if constexpr (LangTraits<L>::kForthFamily) return forth_eval<false>(t, stk, optab, raw);
  else if constexpr (L == kSubleq) return subleq_eval(t, stk, raw);
  else return rsubleq4_eval(t, stk, raw);
}

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
  static constexpr bool kStack = false;
};
template <int L>
struct Stages<L, false> {
  using Lane = ForthFirst<(L == kForthtrivialReset)>;
  template <class W>
  using Warp = ForthWarp<W, (L == kForthtrivialReset)>;
  using Mem = ForthMem;
  static constexpr bool kStack = true;
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

}  // namespace cubff

// Test harness: the machines as a warp runs them, on the host.  Each of the 32
// lanes is a context of its own that runs from one collective (sync, ballot,
// any) to the next, the lanes one after the other in a chosen order: an
// interleaving that CUDA allows, so code that needs lanes to stay in step
// between two syncs gives other results here.  The first stage (and SUBLEQ)
// runs on one lane of the kernels' interleaved words, the other lanes' bytes
// filled with something that must stay.  Test infrastructure only.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <ucontext.h>

#include "interp.cuh"

using namespace cubff;

namespace {

constexpr size_t kStackBytes = 256 << 10;

struct Schedule {
  ucontext_t main, lane[kWarp];
  char *stacks = nullptr;
  bool done[kWarp];
  int kind[kWarp];          // of the collective a lane waits at
  bool value[kWarp];
  uint32_t result, current;
  uint32_t rounds;          // collectives of the last run
  void (*body)(uint32_t);
};
thread_local Schedule g;

void enter() {
  g.body(g.current);
  g.done[g.current] = true;
  swapcontext(&g.lane[g.current], &g.main);
}

// A lane's part of a collective: waits until all lanes are there.
uint32_t collective(uint32_t lane, int kind, bool value) {
  g.kind[lane] = kind;
  g.value[lane] = value;
  swapcontext(&g.lane[lane], &g.main);
  return g.result;
}

// Runs body(lane) for all lanes; false if they do not meet at the same
// collectives.  order: 0 ascending, 1 descending, else another one each time.
bool run_lanes(void (*body)(uint32_t), uint32_t order) {
  g.body = body;
  if (!g.stacks) g.stacks = static_cast<char *>(std::malloc(kWarp * kStackBytes));
  for (uint32_t l = 0; l < kWarp; l++) {
    getcontext(&g.lane[l]);
    g.lane[l].uc_stack.ss_sp = g.stacks + l * kStackBytes;
    g.lane[l].uc_stack.ss_size = kStackBytes;
    g.lane[l].uc_link = nullptr;
    makecontext(&g.lane[l], enter, 0);
    g.done[l] = false;
  }
  for (uint64_t round = 0;; round++) {
    g.rounds = static_cast<uint32_t>(round);
    const uint32_t turn = order < 2 ? (order ? 31 : 0)
                                    : static_cast<uint32_t>(splitmix64(order + round)) & 31;
    uint32_t finished = 0, ballot = 0;
    for (uint32_t q = 0; q < kWarp; q++) {
      const uint32_t l = q ^ turn;
      g.current = l;
      swapcontext(&g.main, &g.lane[l]);
      finished += g.done[l];
    }
    if (finished == kWarp) return true;
    if (finished != 0) return false;
    for (uint32_t l = 0; l < kWarp; l++) {
      if (g.kind[l] != g.kind[0]) return false;
      ballot |= static_cast<uint32_t>(g.value[l]) << l;
    }
    g.result = ballot;
  }
}

// DeviceWarp's interface on such a lane.
struct TurnWarp {
  uint32_t lane;
  template <class T>
  struct Lanes {
    T v;
    T operator()(uint32_t) const { return v; }
  };
  template <class F>
  auto map(F f) const -> Lanes<decltype(f(0u))> {
    return {f(lane)};
  }
  template <class F>
  uint32_t ballot(F f) const {
    return collective(lane, 1, f(lane));
  }
  template <class F>
  bool any(F f) const {
    return collective(lane, 2, f(lane)) != 0;
  }
  template <class F>
  void each(F f) const {
    f(lane);
  }
  void sync() const { collective(lane, 3, false); }
};

struct Counts3 {
  uint32_t ops, raw, mods;
};

// Bytes of `words` that are not lane `lane`'s must be as fill() left them.
template <uint32_t stride>
uint32_t filler(uint32_t w) { return 0x5BD1E995u * (w + stride); }
template <uint32_t stride>
void fill(uint32_t *words) {
  for (uint32_t w = 0; w < stride * kPair / 4; w++) words[w] = filler<stride>(w);
}
template <uint32_t stride>
bool kept(const uint32_t *words, uint32_t lane) {
  for (uint32_t w = 0; w < stride * kPair / 4; w++)
    if (w % stride != lane && words[w] != filler<stride>(w)) return false;
  return true;
}

// What all lanes of the second stage share.
template <int L>
struct Long {
  static thread_local typename Stages<L>::Mem mem;
  static thread_local typename Stages<L>::Lane first;
  static thread_local const uint8_t *optab;
  static thread_local Counts3 counts[kWarp];
  static void lane(uint32_t l) {
    typename Stages<L>::template Warp<TurnWarp> warp(TurnWarp{l}, mem, optab);
    warp.run(first.state());
    counts[l] = {warp.ops(), warp.raw(), warp.mods()};
  }
};
template <int L> thread_local typename Stages<L>::Mem Long<L>::mem;
template <int L> thread_local typename Stages<L>::Lane Long<L>::first;
template <int L> thread_local const uint8_t *Long<L>::optab;
template <int L> thread_local Counts3 Long<L>::counts[kWarp];

// 0: as one program; 1: neighbours' bytes changed; 2: the lanes did not meet;
// 3: the lanes' counts differ.
template <int L, uint32_t stride>
int run_staged(uint8_t *tape, uint32_t lane, uint32_t order, uint32_t steps_on,
               const uint8_t *optab, Counts3 *out) {
  uint32_t tapes[stride * kPair / 4], stacks[stride * kPair / 4];
  fill<stride>(tapes);
  fill<stride>(stacks);
  const LaneWords<stride> t{reinterpret_cast<uint8_t *>(tapes), lane};
  const LaneWords<stride> stk{reinterpret_cast<uint8_t *>(stacks), lane};
  Mask128 cmd{0, 0};
  for (int p = 0; p < kPair; p++) {
    t.set(p, tape[p]);
    mask_assign(cmd, p, optab[tape[p]] < kNull);
  }
  using Lane = typename Stages<L>::Lane;
  Lane &m = Long<L>::first;
  m.begin(t, cmd, optab);
  while (m.status == Lane::kRuns) m.step(t, stk, optab);
  if (m.status == Lane::kJumps) {
    m.resolve(t, optab);
    if constexpr (Stages<L>::kCrowds) {
      typename Lane::Cycle cycle;
      Lane::begin_cycle(cycle);
      for (uint32_t r = 0; r < steps_on && m.status != Lane::kEnds; r++)
        m.step_on(t, stk, optab, cycle);
      m.settle(t, stk, optab);
    }
  }
  if (!kept<stride>(tapes, lane) || !kept<stride>(stacks, lane)) return 1;
  if (m.status == Lane::kEnds) {
    for (int p = 0; p < kPair; p++) tape[p] = static_cast<uint8_t>(t.get(p));
    *out = {m.ops(), m.raw(), m.mods()};
    return 0;
  }
  auto &mem = Long<L>::mem;
  std::memset(&mem, 0xA5, sizeof(mem));
  for (int p = 0; p < kPair; p++) {
    mem.T[p] = static_cast<uint8_t>(t.get(p));
    if constexpr (Stages<L>::kStack) mem.stk[p] = static_cast<uint8_t>(stk.get(p));
  }
  Long<L>::optab = optab;
  if (!run_lanes(&Long<L>::lane, order)) return 2;
  const Counts3 &c = Long<L>::counts[0];
  for (uint32_t l = 1; l < kWarp; l++)
    if (std::memcmp(&Long<L>::counts[l], &c, sizeof(c)) != 0) return 3;
  std::memcpy(tape, mem.T, kPair);
  *out = c;
  return 0;
}

template <bool kRelative4, uint32_t stride>
int run_subleq(uint8_t *tape, uint32_t lane, Counts3 *out) {
  uint32_t tapes[stride * kPair / 4], snaps[stride * kPair / 4];
  fill<stride>(tapes);
  fill<stride>(snaps);
  const LaneWords<stride> t{reinterpret_cast<uint8_t *>(tapes), lane};
  const LaneWords<stride> snap{reinterpret_cast<uint8_t *>(snaps), lane};
  for (int p = 0; p < kPair; p++) t.set(p, tape[p]);
  SubleqMachine<kRelative4> m;
  m.begin();
  while (!m.step(t, snap)) {
  }
  for (int p = 0; p < kPair; p++) tape[p] = static_cast<uint8_t>(t.get(p));
  *out = {m.ops(), m.raw(), m.mods};
  return kept<stride>(tapes, lane) && kept<stride>(snaps, lane) ? 0 : 1;
}

template <int L>
int run_lang(uint32_t stride, uint8_t *tape, uint32_t lane, uint32_t order, uint32_t steps_on,
             Counts3 *out) {
  uint8_t optab[256];
  for (int c = 0; c < 256; c++) optab[c] = op_of(L, c);
  lane %= stride;
  if constexpr (L == kSubleq || L == kRsubleq4) {
    return stride == 16 ? run_subleq<(L == kRsubleq4), 16>(tape, lane, out)
                        : run_subleq<(L == kRsubleq4), 32>(tape, lane, out);
  } else {
    return stride == 8    ? run_staged<L, 8>(tape, lane, order, steps_on, optab, out)
           : stride == 16 ? run_staged<L, 16>(tape, lane, order, steps_on, optab, out)
                          : run_staged<L, 32>(tape, lane, order, steps_on, optab, out);
  }
}

}  // namespace

// Collectives (syncs and votes) of the last run's second stage: its work, on
// every lane alike.
extern "C" uint32_t lanes_rounds() { return g.rounds; }


// Evaluates a tape in place, on lane `lane` of words interleaved by `stride`
// (8, 16 or 32); of a program that goes on, steps_on more steps on the lane, then
// the rest with the lanes taking turns in `order`.
extern "C" int lanes_evaluate(int lang, uint8_t *tape, uint32_t stride, uint32_t lane,
                              uint32_t order, uint32_t steps_on, uint32_t *ops, uint32_t *raw, uint32_t *changed) {
  Counts3 c{};
  int st = -1;
  switch (lang) {
    case kBff: st = run_lang<kBff>(stride, tape, lane, order, steps_on, &c); break;
    case kBffNoheads: st = run_lang<kBffNoheads>(stride, tape, lane, order, steps_on, &c); break;
    case kBffNoheads4bit: st = run_lang<kBffNoheads4bit>(stride, tape, lane, order, steps_on, &c); break;
    case kBffPerm: st = run_lang<kBffPerm>(stride, tape, lane, order, steps_on, &c); break;
    case kBff8: st = run_lang<kBff8>(stride, tape, lane, order, steps_on, &c); break;
    case kBff8Noheads: st = run_lang<kBff8Noheads>(stride, tape, lane, order, steps_on, &c); break;
    case kBffSelfmove: st = run_lang<kBffSelfmove>(stride, tape, lane, order, steps_on, &c); break;
    case kForth: st = run_lang<kForth>(stride, tape, lane, order, steps_on, &c); break;
    case kForthcopy: st = run_lang<kForthcopy>(stride, tape, lane, order, steps_on, &c); break;
    case kForthtrivial: st = run_lang<kForthtrivial>(stride, tape, lane, order, steps_on, &c); break;
    case kForthtrivialReset: st = run_lang<kForthtrivialReset>(stride, tape, lane, order, steps_on, &c); break;
    case kSubleq: st = run_lang<kSubleq>(stride, tape, lane, order, steps_on, &c); break;
    case kRsubleq4: st = run_lang<kRsubleq4>(stride, tape, lane, order, steps_on, &c); break;
  }
  *ops = c.ops;
  *raw = c.raw;
  *changed = c.mods != 0;
  return st;
}

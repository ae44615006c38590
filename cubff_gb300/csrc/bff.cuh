// bff.cuh — the BFF family interpreters (bff, bff_noheads, bff_noheads_4bit,
// bff_perm, bff8, bff8_noheads, bff_selfmove).
//
// Semantics: Evaluate (bff.inc.h:356-389), InitialState (bff.inc.h:269-283),
// EvaluateOne: default (bff.inc.h:289-349), bff8 / bff8_noheads (bff8.cu:23-65),
// bff_selfmove (bff_selfmove.cu:47-98).  The op of a byte comes from the
// language's table (optab, BffOp values).
//
// Two machines that a program runs on in turn:
//  * BffLane, one pair per lane: runs a program until it ends or first jumps
//    (most random programs never do), and on to its end where most of a warp's
//    programs jump (bff8, bff8_noheads: soups of self-replicators);
//  * BffWarp, one pair per warp, which takes over from there.
#pragma once

#include "coop.cuh"
#include "languages.cuh"

namespace cubff {

enum BffLogic { kLogicScan, kLogicJump8, kLogicSelfmove };

// Where a program stands, handed from one machine to the next.
struct BffState {
  int q;             // position of the command to execute
  int h0, h1;        // heads
  uint32_t i, n;     // raw steps before q's command (the no-ops before it included: the
                     // reference counts each as a step and a skip); commands executed,
                     // which is the reference's op count
  uint32_t mods;     // writes that changed a byte
};

// What a lane's cycle check keeps of a program: the state at a taken backward
// jump (q -1: none yet), on Brent's schedule (cycle.cuh).
struct BffCycle {
  int q, h0, h1;
  uint32_t i, n, mods, power, lam;
};

// The forward part of a program on one lane.  The lanes of a warp are at
// different commands, so a step is one straight line of instructions for all
// of them: head moves and value writes all computed and selected.  S marks
// the positions that hold, or once held, a command (a write only ever sets
// bits; a command overwritten by a no-op costs a step that counts no op), so
// a run of no-ops is crossed by finding the next one.
template <bool kHeads, int kLogic, uint32_t kNullMask>
struct BffLane {
  using Cycle = BffCycle;
  enum Status : uint32_t { kRuns, kEnds, kJumps };
  BffState st;
  uint32_t status;
  uint32_t c;         // op of the command at q
  uint32_t v0, v1;    // bytes under the heads
  Mask128 S;

  // cmd_mask: bit p set iff tape byte p is a command (op < kNull).
  template <class Tape>
  __host__ __device__ __forceinline__ void begin(const Tape t, Mask128 cmd_mask,
                                                 const uint8_t *__restrict__ optab) {
    S = cmd_mask;
    st.h0 = kHeads ? t.get(0) & (kPair - 1) : 0;  // no heads: 2 * kSingleTapeSize, masked
    st.h1 = kHeads ? t.get(1) & (kPair - 1) : 0;
    st.i = st.n = st.mods = 0;
    fetch(t, optab, kHeads ? 2 : 0);
  }

  // Moves on to the command at or after position p.
  template <class Tape>
  __host__ __device__ __forceinline__ void fetch(const Tape t,
                                                 const uint8_t *__restrict__ optab, int p) {
    v0 = t.get(st.h0);
    v1 = t.get(st.h1);
    st.q = mask_next(S, p);
    st.i += static_cast<uint32_t>(st.q - p);
    c = optab[t.get(st.q & (kPair - 1))];
    const bool zero = (v0 & kNullMask) == 0;
    const bool jumps = c == kLoopStart ? zero : c == kLoopEnd && !zero;
    status = st.q >= kPair ? kEnds : jumps ? kJumps : kRuns;
  }

  // One command that does not jump (fewer than kPair run, so the step limit is
  // never reached).
  template <class Tape>
  __host__ __device__ __forceinline__ void step(const Tape t, const Tape,
                                                const uint8_t *__restrict__ optab) {
    act(t, optab);
    fetch(t, optab, st.q + 1);
  }
  // What the command at q does but for a jump.
  template <class Tape>
  __host__ __device__ __forceinline__ void act(const Tape t, const uint8_t *__restrict__ optab) {
    st.h0 = (st.h0 + (c == kInc0) - (c == kDec0)) & (kPair - 1);
    st.h1 = (st.h1 + (c == kInc1 || (kLogic == kLogicSelfmove && c == kCopy10)) - (c == kDec1)) &
            (kPair - 1);
    const bool to1 = c == kCopy01, from1 = c == kCopy10;
    const uint32_t v = ((from1 ? v1 : v0) + (c == kPlus) - (c == kMinus)) & 0xFF;
    const uint32_t o = to1 ? v1 : v0;
    if (c - kPlus < 4u && v != o) {
      const int a = to1 ? st.h1 : st.h0;
      t.set(a, v);
      st.mods++;
      if (optab[v] < kNull) mask_assign(S, a, true);
    }
    st.n += c < kNull;
    st.i++;
  }

  // A taken ']' with no '[' before it ends the program (bff8: one that would
  // jump off the tape): tells that from a jump that goes on.
  template <class Tape>
  __host__ __device__ __forceinline__ void resolve(const Tape t,
                                                   const uint8_t *__restrict__ optab) {
    if (c != kLoopEnd) return;
    if (kLogic == kLogicJump8) {
      if (st.q >= 8) return;
    } else {
      for (int b = mask_prev(S, st.q - 1); b >= 0; b = mask_prev(S, b - 1))
        if (optab[t.get(b)] == kLoopStart) return;
    }
    st.n++;
    st.i++;
    status = kEnds;
  }

  __host__ __device__ __forceinline__ static void begin_cycle(BffCycle &y) {
    y.q = -1;
    y.power = 1;
    y.lam = 0;
  }
  // For a program that goes on: the command at q, which may jump; kEnds when it was
  // the program's last.
  template <class Tape>
  __host__ __device__ __forceinline__ void step_on(const Tape t, const Tape,
                                                   const uint8_t *__restrict__ optab,
                                                   BffCycle &y) {
    static_assert(kLogic == kLogicJump8);  // (jumps that need no match)
    const int q = st.q, from = status != kJumps ? q : c == kLoopStart ? q + 8 : q - 8;
    act(t, optab);
    if (from < 0 || from >= kPair) {
      status = kEnds;
      return;
    }
    fetch(t, optab, from + 1);
    if (from < q && status != kEnds && st.i < kStepLimit) visit(y);
    if (st.i >= kStepLimit) status = kEnds;
  }
  // On to a command, for the warp to go on from.
  template <class Tape>
  __host__ __device__ __forceinline__ void settle(const Tape t, const Tape stk,
                                                  const uint8_t *__restrict__ optab) {
    while (status == kRuns && c >= kNull) {
      step(t, stk, optab);
      if (st.i >= kStepLimit) status = kEnds;
    }
  }
  __host__ __device__ __forceinline__ void visit(BffCycle &y) {
    if (st.q == y.q && st.h0 == y.h0 && st.h1 == y.h1 && st.mods == y.mods) {
      const uint32_t len = st.i - y.i, k = (kStepLimit - st.i) / len;
      st.i += k * len;
      st.n += k * (st.n - y.n);
    }
    if (++y.lam == y.power) {
      y.q = st.q;
      y.h0 = st.h0;
      y.h1 = st.h1;
      y.i = st.i;
      y.n = st.n;
      y.mods = st.mods;
      y.power <<= 1;
      y.lam = 0;
    }
  }

  __host__ __device__ __forceinline__ const BffState &state() const { return st; }
  __host__ __device__ __forceinline__ uint32_t ops() const { return st.n; }
  __host__ __device__ __forceinline__ uint32_t raw() const {
    return st.i < kStepLimit ? st.i : kStepLimit;
  }
  __host__ __device__ __forceinline__ uint32_t mods() const { return st.mods; }
};

// Shared memory of one warp's BffWarp.
struct alignas(16) BffMem {
  uint8_t T[kPair];      // the pair tape
  uint8_t snap[kPair];   // its snapshot at a taken ']'
  uint8_t top[kPair];    // its snapshot at the top of a loop
  uint16_t E[kPair];     // op | position of the next command << 8 (kPair: none)
  uint8_t D[kPair];      // '[' minus ']' up to and including the position, mod 256
  uint16_t M[kPair];     // bracket matches: position | straight << 7, kNone or kUnknown
  uint32_t P[8];         // micro-ops of the compiled loop
  uint8_t X[kWarp];      // one byte per lane
};
static_assert(sizeof(BffMem) % 16 == 0, "BffMem");

// One pair on a whole warp, from its first jump on.
//
// What bounds it: the chain of dependent instructions of one program (~4.4
// cycles each), so the lanes are used to make that chain short:
//  * decoding (the ops, the next command after every position, bracket
//    depths) is done for all 128 positions at once.  A write that changes a
//    byte's op only widens the range [dlo, dhi] of positions changed since;
//    what is used of the decode must lie outside it, else it is redone (a
//    replicator writes the other program's bytes while it runs its own);
//  * a bracket's match is found on bit masks, or over the depths when other
//    brackets lie between, and kept;
//  * a loop [ ... ] without inner brackets is compiled to micro-ops (the net
//    head moves up to the next '+' / '-' run, copy or the ']', and that
//    command, at most 8) and counts once per iteration.  Bodies with at most
//    one copy run up to 32 iterations at a time, one per lane; a body that only
//    counts the tested byte is solved; others go micro-op by micro-op.  A write
//    into the loop's own code leaves the loop before the command that does it
//    (a byte changed to another of the same op does not count);
//  * exact cycle fast-forward at other taken ']'s, on Brent's schedule
//    (cycle.cuh): the state is (position, heads, tape), and the tape is
//    compared with a snapshot four bytes per lane.  Head 1 may differ when no
//    copy used it since the snapshot (every ']' tests the byte under head 0):
//    control flow depends only on the rest, so the segment since the snapshot
//    repeats with that head shifted by the same amount each time; k
//    repetitions advance i, n and the head by k times the segment's;
//  * a compiled loop moves its heads by the same net amounts each iteration,
//    so they are back after `period` iterations (at most 128).  As many
//    iterations in a row without a changed byte and without leaving mean that
//    none will ever come: the loop runs to the step limit.
//
// Uniform stores are made by every lane (the same value to the same place) after
// a sync: by then all lanes have read what the store changes and made the one
// before, so a lane that is ahead or behind reads nothing else, and every lane
// reads at least its own.  Lane-wise stores are between two syncs.
template <class W, int kLogic, uint32_t kNullMask>
struct BffWarp {
  static constexpr uint32_t kSettle = 8;  // micro-op loop iterations before the first visit
  // Micro-ops: the net moves mod 128 at bits 0 and 8, act at 16, and what kAdd
  // adds (a run of '+' or '-'), mod 256, at 24.
  enum Act : uint32_t { kAdd, kTo0, kTest, kTo1 };  // (bit 0: a copy; both bits: to head 1)
  enum Kind : uint32_t { kGeneric, kCopyOne, kCount };
  static constexpr int kEnd = -1, kRedo = -2;
  static constexpr uint32_t kNone = 0x100, kUnknown = 0x200;

  const W w;
  BffMem &m;
  const uint8_t *const optab;
  BffState st;
  uint32_t v0, v1;    // bytes under the heads (not kept up to date in loops)
  int dlo, dhi;       // positions whose op changed since the decode (none: dlo > dhi)
  uint32_t open[4], close[4];  // brackets, 32 positions a word
  bool used1;         // a copy used head 1 since the snapshot
  // The compiled loop: '[' at ls, ']' at le (-1: none), its micro-ops (m.P),
  // the commands of an iteration, the net moves, its period and kind.
  int ls, le, net0, net1;
  uint32_t lcmds, period, kind;
  bool copies;        // it has copies
  // Taken ']'s still to step through one by one after a loop wrote into its
  // own code at once, and as many the next time: so the cycle check sees them.
  uint32_t hold, backoff;
  uint32_t iters;     // iterations done in it
  // Snapshot taken at a taken ']'.
  int s_key, s_h0, s_h1;
  uint32_t s_i, s_n, s_mods, s_power, s_lam;

  __host__ __device__ __forceinline__ BffWarp(W warp, BffMem &mem, const uint8_t *table)
      : w(warp), m(mem), optab(table) {}

  __host__ __device__ __forceinline__ uint32_t word(const uint8_t *a, uint32_t l) const {
    return reinterpret_cast<const uint32_t *>(a)[l];
  }

  // Ops, next commands, brackets and depths of all positions.
  __host__ __device__ __forceinline__ void decode() {
    if (dlo <= le && dhi >= ls) le = -1;
    w.sync();
    // Matches stay where no op between the two brackets changed.
    w.each([&](uint32_t l) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t r = m.M[32 * k + l];
        const bool stays = r < kNone && clean(static_cast<int>(32 * k + l), static_cast<int>(r & 127));
        m.M[32 * k + l] = static_cast<uint16_t>(stays ? r : kUnknown);
      }
    });
    dlo = kPair;
    dhi = -1;
    const auto op0 = w.map([&](uint32_t l) { return uint32_t(optab[m.T[l]]); });
    const auto op1 = w.map([&](uint32_t l) { return uint32_t(optab[m.T[32 + l]]); });
    const auto op2 = w.map([&](uint32_t l) { return uint32_t(optab[m.T[64 + l]]); });
    const auto op3 = w.map([&](uint32_t l) { return uint32_t(optab[m.T[96 + l]]); });
    auto op = [&](int k, uint32_t l) {
      return k == 0 ? op0(l) : k == 1 ? op1(l) : k == 2 ? op2(l) : op3(l);
    };
    uint32_t cmd[4], above[4];
    int sum[4], total = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      cmd[k] = w.ballot([&](uint32_t l) { return op(k, l) < kNull; });
      open[k] = w.ballot([&](uint32_t l) { return op(k, l) == kLoopStart; });
      close[k] = w.ballot([&](uint32_t l) { return op(k, l) == kLoopEnd; });
      sum[k] = total;
      total += popc32(open[k]) - popc32(close[k]);
    }
    above[3] = kPair;
#pragma unroll
    for (int k = 2; k >= 0; k--) above[k] = cmd[k + 1] ? 32 * k + 32 + low32(cmd[k + 1]) : above[k + 1];
    w.each([&](uint32_t l) {
      const uint32_t upto = ~0u >> (31 - l);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        m.D[32 * k + l] =
            static_cast<uint8_t>(sum[k] + popc32(open[k] & upto) - popc32(close[k] & upto));
        const uint32_t x = cmd[k] & ~upto;
        m.E[32 * k + l] =
            static_cast<uint16_t>(op(k, l) | (x ? 32 * k + low32(x) : above[k]) << 8);
      }
    });
    w.sync();
  }

  // Ops of positions lo..hi may have changed.
  __host__ __device__ __forceinline__ void changed_op(int lo, int hi) {
    dlo = lo < dlo ? lo : dlo;
    dhi = hi > dhi ? hi : dhi;
  }

  // Writes v over o != v at position p.
  __host__ __device__ __forceinline__ void write(int p, uint32_t o, uint32_t v) {
    w.sync();
    m.T[p] = static_cast<uint8_t>(v);
    st.mods++;
    if (optab[v] != optab[o]) changed_op(p, p);
  }

  // No op between a and b (in either order) changed since the decode.
  __host__ __device__ __forceinline__ bool clean(int a, int b) const {
    return dlo > (a > b ? a : b) || dhi < (a > b ? b : a);
  }

  // The match of the bracket at q (op c): position, | 128 when no brackets lie
  // between; kNone when there is none; kUnknown when ops must be decoded again
  // first.
  __host__ __device__ __forceinline__ uint32_t match(int q, uint32_t c) {
    uint32_t r = m.M[q];
    if (r == kUnknown) r = search(q, c);
    const bool stale = dlo <= dhi && (r == kNone || !clean(q, static_cast<int>(r & 127)));
    return stale ? kUnknown : r;
  }

  // One set bit at or beyond which a search goes on: word k of the positions
  // above q (fwd) or below it.
  __host__ __device__ __forceinline__ static uint32_t beyond(int k, int q, bool fwd) {
    const uint32_t upto = ~0u >> (31 - (q & 31));
    return k == (q >> 5) ? (fwd ? ~upto : upto >> 1) : (k > (q >> 5)) == fwd ? ~0u : 0u;
  }
  // The first of the masked positions above q, or the last below it; -1.
  __host__ __device__ __forceinline__ static int nearest(uint32_t x0, uint32_t x1, uint32_t x2,
                                                         uint32_t x3, bool fwd) {
    if (fwd) return x0 ? low32(x0) : x1 ? 32 + low32(x1) : x2 ? 64 + low32(x2) : x3 ? 96 + low32(x3) : -1;
    return x3 ? 96 + high32(x3) : x2 ? 64 + high32(x2) : x1 ? 32 + high32(x1) : x0 ? high32(x0) : -1;
  }
  // match(), searched for and kept.
  __host__ __device__ __forceinline__ uint32_t search(int q, uint32_t c) {
    const bool fwd = c == kLoopStart;
    uint32_t far[4];
#pragma unroll
    for (int k = 0; k < 4; k++) far[k] = beyond(k, q, fwd);
    const int near = nearest((open[0] | close[0]) & far[0], (open[1] | close[1]) & far[1],
                             (open[2] | close[2]) & far[2], (open[3] | close[3]) & far[3], fwd);
    uint32_t r = kNone;
    if (near >= 0) {
      if ((m.E[near] & 15u) != c) {  // the next bracket is the match
        r = static_cast<uint32_t>(near) | 128u;
      } else {
        // Forward: the first ']' that brings the depth below that at q; back:
        // the last '[' that brings it one above.
        const uint32_t want = (m.D[q] + (fwd ? 0xFFu : 1u)) & 0xFF;
        uint32_t hit[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          hit[k] = far[k] & (fwd ? close[k] : open[k]) &
                   w.ballot([&](uint32_t l) { return m.D[32 * k + l] == want; });
        const int b = nearest(hit[0], hit[1], hit[2], hit[3], fwd);
        if (b >= 0) r = static_cast<uint32_t>(b);
      }
    }
    w.sync();
    m.M[q] = static_cast<uint16_t>(r);
    if (r != kNone) m.M[r & 127] = static_cast<uint16_t>(static_cast<uint32_t>(q) | (r & 128));
    return r;
  }

  // At a taken ']', in the state named by key (where execution goes on).
  __host__ __device__ __forceinline__ void visit(int key) {
    if (key == s_key && st.h0 == s_h0 && (!used1 || st.h1 == s_h1) && st.i < kStepLimit &&
        (st.mods == s_mods ||
         !w.any([&](uint32_t l) { return word(m.T, l) != word(m.snap, l); }))) {
      const uint32_t len = st.i - s_i;
      const uint32_t k = (kStepLimit - st.i) / len;
      st.i += k * len;
      st.n += k * (st.n - s_n);
      if (st.h1 != s_h1) {
        st.h1 = (st.h1 + static_cast<int>(k) * (st.h1 - s_h1)) & (kPair - 1);
        v1 = m.T[st.h1];
      }
    }
    if (++s_lam == s_power) {
      s_key = key;
      s_h0 = st.h0;
      s_h1 = st.h1;
      s_i = st.i;
      s_n = st.n;
      s_mods = st.mods;
      s_power <<= 1;
      s_lam = 0;
      used1 = false;
      w.sync();
      w.each([&](uint32_t l) {
        reinterpret_cast<uint32_t *>(m.snap)[l] = word(m.T, l);
      });
      w.sync();
    }
  }

  // Compiles the loop from '[' at s to ']' at e, with no brackets between and
  // no op changed since the decode; false when it has too many micro-ops.
  __host__ __device__ __forceinline__ bool compile(int s, int e) {
    w.sync();
    le = -1;
    int k = 0, d0 = 0, d1 = 0, m0 = 0, m1 = 0;
    uint32_t cmds = 1, last = kNoop, u = 0, first = 0;
    copies = false;
    for (int p = s;;) {
      p = m.E[p] >> 8;
      const uint32_t op = p < e ? m.E[p] & 15u : static_cast<uint32_t>(kLoopEnd);
      if (op >= kDec0) {
        cmds++;
        if (op <= kInc0) d0 += op == kInc0 ? 1 : -1;
        else d1 += op == kInc1 ? 1 : -1;
        last = kNoop;
        continue;
      }
      if (op != kLoopEnd) cmds++;
      if (op == last) {  // a repeated copy changes nothing more; a run of '+' or '-' adds up
        if (op <= kMinus) {
          u += op == kPlus ? 1u << 24 : ~0u << 24;
          m.P[k - 1] = u;
        }
        continue;
      }
      if (k == 8) return false;
      m0 += d0;
      m1 += d1;
      const uint32_t act = op == kLoopEnd ? kTest : op == kCopy01 ? kTo1 : op == kCopy10 ? kTo0 : kAdd;
      u = static_cast<uint32_t>((d0 & (kPair - 1)) | (d1 & (kPair - 1)) << 8) | act << 16 |
          (op == kPlus ? 1u << 24 : op == kMinus ? ~0u << 24 : 0u);
      m.P[k] = u;
      if (k == 0) first = act;
      k++;
      if (op == kLoopEnd) break;
      d0 = d1 = 0;
      last = op;
      copies |= act != kAdd;
      if (kLogic == kLogicSelfmove && op == kCopy10) {
        d1 = 1;
        last = kNoop;
      }
    }
    w.sync();
    ls = s;
    le = e;
    net0 = m0;
    net1 = m1;
    lcmds = cmds;
    const uint32_t moved = static_cast<uint32_t>(m0 | (copies ? m1 : 0)) | kPair;
    period = static_cast<uint32_t>(kPair >> low32(moved));
    kind = k == 1 || (k == 2 && first != kAdd)    ? kCopyOne
           : k == 2 && m0 == 0 && (u & 0x7F) == 0 ? kCount
                                                  : kGeneric;
    return true;
  }

  // The loop changes nothing more and never ends: runs it to the step limit.
  __host__ __device__ __forceinline__ int run_out() {
    const uint32_t len = static_cast<uint32_t>(le - ls), k = (kStepLimit - st.i) / len;
    st.i += k * len;
    st.n += k * lcmds;
    const int end = ls + 1 + static_cast<int>(kStepLimit - st.i);
    for (int p = m.E[ls] >> 8; p < end; p = m.E[p] >> 8) st.n++;
    st.i = kStepLimit;
    return kEnd;
  }

  // The command at hand (the body's left-th that is no move) would write into
  // the loop's code: leaves the loop, the heads moved, before it.
  __host__ __device__ __forceinline__ int bail(int left) {
    if (iters < 2) {
      hold = backoff;
      if (backoff < 64) backoff *= 2;
    } else {
      backoff = 4;
    }
    // Found as compile() counts them.
    uint32_t last = kNoop;
    int p = m.E[ls] >> 8;
    for (; p < le; p = m.E[p] >> 8) {
      const uint32_t op = m.E[p] & 15;
      if (op < kDec0 && op != last && --left == 0) break;
      last = op >= kDec0 || (kLogic == kLogicSelfmove && op == kCopy10)
                 ? static_cast<uint32_t>(kNoop) : op;
      st.n++;
    }
    st.i += static_cast<uint32_t>(p - 1 - ls);
    return p - 1;
  }

  // Runs the compiled loop from its top until it ends, is left or reaches the
  // step limit.  A whole iteration fits in the limit on entry.  This and the
  // functions that run commands return the position after which execution
  // goes on (raw steps through it counted), or kEnd.
  __host__ __device__ __forceinline__ int loop() {
    iters = 0;
    used1 |= copies;
    const uint32_t len = static_cast<uint32_t>(le - ls);
    if (kind == kCopyOne) return loop_copy(len);
    if (kind == kCount && (st.h0 < ls || st.h0 > le)) return loop_count(len);
    return loop_generic(len);
  }

  // At most one copy.  Lane j is iteration j: it reads from src + j * ds,
  // writes to dst + j * dd, and the ']' reads test + j * net0.  Iterations are
  // cut where one would read what an earlier one of the same batch changed: `most`
  // after the first that changes a byte.  (Heads that part ways, as in a copy
  // backwards, leave just that one, but once copied nothing changes any more: 64
  // epochs of 2^17 bff_noheads_4bit programs evolved for 4096 58 ms, 96 with one
  // iteration at a time throughout.)
  __host__ __device__ __forceinline__ int loop_copy(uint32_t len) {
    const uint32_t u = m.P[0], act = (u >> 16) & 3;
    const bool to1 = act == kTo1;
    const int a0 = copies ? static_cast<int>(u & 127) : net0;
    const int a1 = static_cast<int>((u >> 8) & 127);
    const int ds = act == kTo0 ? net1 : net0, dd = to1 ? net1 : net0;
    uint32_t most = kWarp;
    if (copies) {
      // Iterations that lie apart by so many read what the earlier one wrote.
      const int x0 = st.h0 + a0, x1 = st.h1 + a1;
      const int off_s = act == kTo0 ? x1 - x0 : x0 - x1;
      const int off_t = st.h0 + net0 - (to1 ? x1 : x0);
      if (dd == net0 && dd == ds && (dd == 1 || dd == -1)) {
        const uint32_t js = static_cast<uint32_t>(-off_s * dd) & (kPair - 1);
        const uint32_t jt = static_cast<uint32_t>(-off_t * dd) & (kPair - 1);
        if (js - 1 < most - 1) most = js;
        if (jt - 1 < most - 1) most = jt;
      } else if (dd != 0) {
        const uint32_t bad = w.ballot([&](uint32_t l) {
          const int j = static_cast<int>(l);
          bool b = ((dd * j) & (kPair - 1)) == 0;                      // the same byte written again
          if (ds == dd) b |= ((off_s + ds * j) & (kPair - 1)) == 0;    // a written byte copied on
          if (net0 == dd) b |= ((off_t + dd * j) & (kPair - 1)) == 0;  // a written byte tested later
          if ((ds != dd && ds != 0) || (net0 != dd && net0 != 0)) b = true;
          return b && j > 0;
        });
        if (bad) most = static_cast<uint32_t>(low32(bad));
      }
    }
    uint32_t quiet = 0;
    while (true) {
      uint32_t room = kWarp;
      if (st.i + kWarp * len > kStepLimit) room = (kStepLimit - st.i) / len;
      const int t0 = st.h0 + net0, s0 = act == kTo0 ? st.h1 + a1 : st.h0 + a0;
      const int w0 = to1 ? st.h1 + a1 : st.h0 + a0;
      uint32_t cut = room;
      const auto at = w.map([&](uint32_t l) { return (w0 + dd * static_cast<int>(l)) & (kPair - 1); });
      const auto x = w.map([&](uint32_t l) {
        return uint32_t(m.T[(s0 + ds * static_cast<int>(l)) & (kPair - 1)]);
      });
      const auto y = w.map([&](uint32_t l) { return uint32_t(m.T[at(l)]); });
      const auto z = w.map([&](uint32_t l) {
        const int p = (t0 + net0 * static_cast<int>(l)) & (kPair - 1);
        return copies && p == at(l) ? x(l) : uint32_t(m.T[p]);
      });
      uint32_t changed = copies ? w.ballot([&](uint32_t l) { return x(l) != y(l); }) : 0u;
      if (changed != 0 && low32(changed) + most < cut) cut = low32(changed) + most;
      if (copies && (changed != 0 || dd == 0)) {
        if (dd == 0) {
          // One byte written over and over: cut before an iteration that reads
          // it; iteration j > 0 finds what j - 1 wrote.
          if (ds != 0) {
            const uint32_t self = w.ballot([&](uint32_t l) {
              return l > 0 && ((s0 + ds * static_cast<int>(l) - w0) & (kPair - 1)) == 0;
            });
            if (self && static_cast<uint32_t>(low32(self)) < cut) cut = low32(self);
          }
          w.sync();
          w.each([&](uint32_t l) { m.X[l] = static_cast<uint8_t>(x(l)); });
          w.sync();
          changed = (changed & 1) |
                    w.ballot([&](uint32_t l) { return l > 0 && m.X[l - 1] != x(l); });
        } else if (net0 == 0) {
          // One byte tested throughout: cut after the iteration that writes it.
          const uint32_t hits = w.ballot([&](uint32_t l) { return at(l) == (t0 & (kPair - 1)); });
          if (hits && static_cast<uint32_t>(low32(hits)) + 1 < cut) cut = low32(hits) + 1;
        }
        const uint32_t code = changed == 0 ? 0u : changed & w.ballot([&](uint32_t l) {
          return static_cast<uint32_t>(at(l) - ls) <= len;
        });
        if (code) {
          // A change of the loop's code is one of its ops.
          const uint32_t ops = code & w.ballot([&](uint32_t l) {
            return optab[x(l)] != optab[dd == 0 && l > 0 ? m.X[l - 1] : y(l)];
          });
          const uint32_t first = ops ? static_cast<uint32_t>(low32(ops)) : kWarp;
          if (first < cut) cut = first;
          if (cut == 0) {
            st.h0 = (st.h0 + a0) & (kPair - 1);
            st.h1 = (st.h1 + a1) & (kPair - 1);
            return bail(1);
          }
        }
      }
      uint32_t zero = w.ballot([&](uint32_t l) { return (z(l) & kNullMask) == 0; });
      const uint32_t within = ~0u >> (32 - cut);
      zero &= within;
      if (zero) cut = low32(zero) + 1;
      changed &= zero ? ~0u >> (32 - cut) : within;
      if (changed) {
        w.sync();
        // (One byte: the last iteration's value stays.)
        const uint32_t ops = w.ballot([&](uint32_t l) {
          if (dd == 0 ? l + 1 != cut : !((changed >> l) & 1)) return false;
          m.T[at(l)] = static_cast<uint8_t>(x(l));
          return optab[x(l)] != optab[y(l)];
        });
        w.sync();
        if (ops) {  // the range of the changed positions, which go from the first lane's by dd
          const int a = (w0 + dd * low32(ops)) & (kPair - 1), b = a + dd * (high32(ops) - low32(ops));
          if (b >= 0 && b < kPair) changed_op(a < b ? a : b, a < b ? b : a);
          else changed_op(0, kPair - 1);
        }
        st.mods += popc32(changed);
        quiet = cut - 1 - high32(changed);
      } else {
        quiet += cut;
      }
      st.h0 = (st.h0 + net0 * static_cast<int>(cut)) & (kPair - 1);
      st.h1 = (st.h1 + net1 * static_cast<int>(cut)) & (kPair - 1);
      st.i += cut * len;
      st.n += cut * lcmds;
      iters += cut;
      if (zero) return le;
      if (quiet >= period) return run_out();
      if (st.i + len > kStepLimit) return ls;
    }
  }

  // One run of '+' or '-' on the tested byte, outside the loop's code: the
  // iterations until it is zero (or all that the step limit allows) at once.
  __host__ __device__ __forceinline__ int loop_count(uint32_t len) {
    const uint32_t d = m.P[0] >> 24;
    const uint32_t o = m.T[st.h0];
    const uint32_t room = (kStepLimit - st.i) / len;
    uint32_t k = 0;
    bool found = false;
    while (k < room && k < 256 && !found) {  // the byte's values repeat after 256
      const uint32_t zero = w.ballot([&](uint32_t l) {
        return k + l < room && ((o + (k + l + 1) * d) & kNullMask) == 0;
      });
      found = zero != 0;
      k += found ? low32(zero) + 1 : kWarp;
    }
    if (!found) k = room;
    const uint32_t v = (o + k * d) & 0xFF;
    if (v != o) write(st.h0, o, v);
    st.i += k * len;
    st.n += k * lcmds;
    st.h1 = (st.h1 + static_cast<int>(k) * net1) & (kPair - 1);
    return found ? le : ls;
  }

  // Whether micro-op u changes the op of a byte from o to v, or of one passed on
  // the way of a run.
  __host__ __device__ __forceinline__ bool code_changes(uint32_t u, uint32_t o, uint32_t v) const {
    const bool down = u >> 31, copy = (u >> 16) & 1;
    const uint32_t r = copy ? 1u : down ? 256 - (u >> 24) : u >> 24;
    return r > kWarp || w.any([&](uint32_t l) {
      const uint32_t x = copy ? v : down ? o - l - 1 : o + l + 1;
      return l < r && optab[x & 0xFF] != optab[o];
    });
  }

  // Micro-op by micro-op.  The cycle check (on a snapshot of its own) runs
  // whenever the heads are back where they were after the first kSettle
  // iterations.
  __host__ __device__ __forceinline__ int loop_generic(uint32_t len) {
    const uint32_t spacing = period < kSettle ? kSettle : period;
    uint32_t quiet = 0, until = kSettle, since = 0, power = 0;
    int lo = kPair, hi = -1, from;  // lo..hi: positions written
    while (true) {
      uint32_t u = m.P[0];
      int k = 0;
      do {
        st.h0 = (st.h0 + static_cast<int>(u)) & (kPair - 1);
        st.h1 = (st.h1 + static_cast<int>(u >> 8)) & (kPair - 1);
        const uint32_t b0 = m.T[st.h0], b1 = m.T[st.h1];
        const bool copy = (u >> 16) & 1, to1 = (u >> 17) & 1;
        const uint32_t o = to1 ? b1 : b0;
        const uint32_t v = copy ? (to1 ? b0 : b1) : (b0 + (u >> 24)) & 0xFF;
        const int p = to1 ? st.h1 : st.h0;
        const uint32_t was = u;
        u = m.P[++k];
        if (v != o) {
          if (static_cast<uint32_t>(p - ls) <= len && code_changes(was, o, v)) {
            if (lo <= hi) changed_op(lo, hi);
            return bail(k);
          }
          w.sync();
          m.T[p] = static_cast<uint8_t>(v);
          st.mods++;
          lo = p < lo ? p : lo;
          hi = p > hi ? p : hi;
          quiet = ~0u;
        }
      } while (((u >> 16) & 3) != kTest);
      st.h0 = (st.h0 + static_cast<int>(u)) & (kPair - 1);
      st.h1 = (st.h1 + static_cast<int>(u >> 8)) & (kPair - 1);
      st.i += len;
      st.n += lcmds;
      from = le;
      if ((m.T[st.h0] & kNullMask) == 0) break;
      iters++;
      if (++quiet >= period) {
        from = run_out();
        break;
      }
      if (--until == 0) {
        until = spacing;
        since += spacing;
        if (power != 0 && !w.any([&](uint32_t l) { return word(m.T, l) != word(m.top, l); })) {
          const uint32_t room = (kStepLimit - st.i) / len, skip = room - room % since;
          st.i += skip * len;
          st.n += skip * lcmds;
          st.h1 = (st.h1 + static_cast<int>(skip) * net1) & (kPair - 1);
        }
        if (since >= power * spacing) {  // renewed after 1, 2, 4, ... checks
          power = power ? 2 * power : 1;
          since = 0;
          w.each([&](uint32_t l) { reinterpret_cast<uint32_t *>(m.top)[l] = word(m.T, l); });
        }
      }
      from = ls;
      if (st.i + len > kStepLimit) break;
    }
    if (lo <= hi) changed_op(lo, hi);
    return from;
  }

  // A bracket at q; back: a ']' was taken (and is no compiled loop's).  kRedo,
  // with nothing done, when ops must be decoded again first.
  __host__ __device__ __forceinline__ int bracket(uint32_t c, bool *back) {
    const bool zero = (v0 & kNullMask) == 0, taken = zero == (c == kLoopStart);
    const int q = st.q;
    int from = q;
    uint32_t mt = kNone;
    if (kLogic == kLogicJump8) {
      if (taken) from = c == kLoopStart ? q + 8 : q - 8;
      *back = from < q;
      if (from < 0 || from >= kPair) from = kEnd;
    } else if (c == kLoopStart || taken) {
      mt = match(q, c);
      if (mt == kUnknown) return kRedo;
      if (taken) from = mt == kNone ? kEnd : static_cast<int>(mt & 127);
    }
    st.n++;
    st.i++;
    if (kLogic == kLogicJump8) return from;
    if ((mt & 128) != 0 && (c == kLoopEnd || !zero)) {
      const int b = static_cast<int>(mt & 127), s = c == kLoopStart ? q : b,
                e = c == kLoopStart ? b : q;
      if (hold != 0) hold -= taken;
      else if (((s == ls && e == le) || compile(s, e)) &&
               st.i + static_cast<uint32_t>(e - s) <= kStepLimit)
        return loop();
    }
    *back = taken && c == kLoopEnd;
    return from;
  }

  // A command other than a bracket, at q.
  __host__ __device__ __forceinline__ void command(uint32_t c) {
    st.n++;
    st.i++;
    if (c >= kDec1) {
      st.h1 = (st.h1 + (c == kInc1 ? 1 : -1)) & (kPair - 1);
      v1 = m.T[st.h1];
    } else if (c >= kDec0) {
      st.h0 = (st.h0 + (c == kInc0 ? 1 : -1)) & (kPair - 1);
      v0 = m.T[st.h0];
    } else {
      const bool to1 = c == kCopy01;
      const uint32_t v =
          (c == kPlus ? v0 + 1 : c == kMinus ? v0 - 1 : c == kCopy10 ? v1 : v0) & 0xFF;
      const uint32_t o = to1 ? v1 : v0;
      used1 |= c >= kCopy01;
      if (v != o) {
        write(to1 ? st.h1 : st.h0, o, v);
        if (!to1 || st.h0 == st.h1) v0 = v;
        if (to1 || st.h0 == st.h1) v1 = v;
      }
      if (kLogic == kLogicSelfmove && c == kCopy10) {
        st.h1 = (st.h1 + 1) & (kPair - 1);
        v1 = m.T[st.h1];
      }
    }
  }

  // The state at the start of the program in m.T: at its first command.
  __host__ __device__ __forceinline__ BffState start(bool heads) const {
    const int pc = heads ? 2 : 0;
    int q = kPair;
#pragma unroll
    for (int k = 3; k >= 0; k--) {
      const uint32_t cmd = w.ballot([&](uint32_t l) {
        return static_cast<int>(32 * k + l) >= pc && optab[m.T[32 * k + l]] < kNull;
      });
      if (cmd) q = 32 * k + low32(cmd);
    }
    return {q, heads ? m.T[0] & (kPair - 1) : 0, heads ? m.T[1] & (kPair - 1) : 0,
            static_cast<uint32_t>(q - pc), 0, 0};
  }

  // Runs the program in m.T from state s (at a command) to its end; ops() and
  // raw() are then its op and raw step counts.
  __host__ __device__ __forceinline__ void run(const BffState &s) {
    st = s;
    used1 = true;
    copies = false;
    ls = le = s_key = -1;
    net0 = net1 = 0;
    lcmds = period = kind = iters = hold = 0;
    backoff = 4;
    s_h0 = s_h1 = 0;
    s_i = s_n = s_mods = s_lam = 0;
    s_power = 1;
    dlo = 0;
    dhi = kPair - 1;  // nothing is decoded yet
    v0 = m.T[st.h0];
    v1 = m.T[st.h1];
    if (st.q >= kPair) return;
    int from = kRedo, next = 0;
    bool back = false;
    while (true) {
      // On to the command after `from` (or st.q once more).
      if (from == kRedo || (dlo <= next && dhi > from)) {
        decode();
        if (from != kRedo) next = m.E[from] >> 8;
      }
      if (from != kRedo) {
        st.i += static_cast<uint32_t>(next - from - 1);
        st.q = next;
        if (next >= kPair || st.i >= kStepLimit) return;
        if (back) {
          visit(next);
          if (st.i >= kStepLimit) return;
        }
      }
      const uint32_t en = m.E[st.q], c = en & 15;
      back = false;
      if (c > kLoopEnd) {
        command(c);
        from = st.q;
        next = en >> 8;
      } else {
        from = bracket(c, &back);
        if (from == kEnd) return;
        if (from != kRedo) {
          v0 = m.T[st.h0];
          v1 = m.T[st.h1];
          next = m.E[from] >> 8;
        }
      }
    }
  }

  __host__ __device__ __forceinline__ uint32_t ops() const { return st.n; }
  __host__ __device__ __forceinline__ uint32_t mods() const { return st.mods; }
  __host__ __device__ __forceinline__ uint32_t raw() const {
    return st.i < kStepLimit ? st.i : kStepLimit;
  }
};

}  // namespace cubff

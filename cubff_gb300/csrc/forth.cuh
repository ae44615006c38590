// forth.cuh — the Forth family interpreters (forth, forthcopy, forthtrivial,
// forthtrivial_reset).
//
// Semantics: Stack (forth.inc.h:236-249), EvaluateOne (forth.inc.h:250-373),
// Evaluate (forth.inc.h:379-397); forthtrivial_reset's Reset / ResetIf and its
// Write1 / Copy0 (forthtrivial_reset.cu:58-72, :157-166, :215-223).  The top
// two entries of the 128-byte stack are kept in registers.
//
// Two machines that a program runs on in turn:
//  * ForthFirst, one pair per lane, for a program's first steps (most random
//    programs end in them), and for the rest where most of a warp's programs
//    go on (a soup of self-replicators);
//  * ForthWarp, one pair per warp, which takes over from there.
#pragma once

#include "coop.cuh"
#include "languages.cuh"

namespace cubff {

// Byte i that a reset at position pos writes.
__host__ __device__ __forceinline__ uint8_t reset_byte(uint64_t seed, int pos, uint32_t i) {
  return static_cast<uint8_t>(
      splitmix64(seed * kTape * kTape + static_cast<uint64_t>(pos * kTape) + i));
}
template <class Tape>
static __host__ __device__ __noinline__ void forth_reset(const Tape t, int pos) {
  uint64_t seed = 0;
  for (int i = 0; i < kPair; i++) seed = splitmix64(seed ^ t.get(i));
  for (int i = 0; i < kTape; i++) t.set(i, reset_byte(seed, pos, i));
}
// The seed of a reset on the whole warp, of a tape in 4-byte aligned words: a chain
// of 128 draws, for which the next word is on its way.  (The 64 bytes written are
// then two to a lane.  Soups of forthtrivial_reset that had evolved for 1024 epochs,
// 64 epochs: 2^14 programs 119 ms, 2^17 191 ms; byte by byte on every lane 188 and
// 288, one pair a lane 147 and 187.)
static __host__ __device__ __noinline__ uint64_t reset_seed(const uint8_t *tape) {
  const uint32_t *words = reinterpret_cast<const uint32_t *>(tape);
  uint64_t seed = 0;
  uint32_t next = words[0];
  for (int q = 0; q < kPair / 4; q++) {
    const uint32_t w = next;
    next = words[(q + 1) % (kPair / 4)];
#pragma unroll
    for (int b = 0; b < 4; b++) seed = splitmix64(seed ^ ((w >> (8 * b)) & 0xFF));
  }
  return seed;
}

// Positions written in each half of a tape: [lo, hi] (none: lo > hi).
struct Written {
  int lo0, hi0, lo1, hi1;
  __host__ __device__ __forceinline__ bool none() const { return hi0 < 0 && hi1 < 0; }
  __host__ __device__ __forceinline__ void clear() {
    lo0 = lo1 = kPair;
    hi0 = hi1 = -1;
  }
  __host__ __device__ __forceinline__ void add(int p) {
    if (p < kTape) {
      lo0 = p < lo0 ? p : lo0;
      hi0 = p > hi0 ? p : hi0;
    } else {
      lo1 = p < lo1 ? p : lo1;
      hi1 = p > hi1 ? p : hi1;
    }
  }
  __host__ __device__ __forceinline__ bool meets(int lo, int hi) const {
    return (lo0 <= hi && hi0 >= lo) || (lo1 <= hi && hi1 >= lo);
  }
};
// A warp's tape: all lanes have read before any writes (ForthWarp), and what is
// written is noted.
template <class W>
struct TrackedBytes {
  const W &w;
  uint8_t *s;
  Written &written;
  __host__ __device__ __forceinline__ uint32_t get(int p) const { return s[p & (kPair - 1)]; }
  __host__ __device__ __forceinline__ void set(int p, uint32_t v) const {
    w.sync();
    s[p & (kPair - 1)] = static_cast<uint8_t>(v);
    written.add(p);
  }
};
// A warp's stack.
template <class W>
struct StackBytes {
  const W &w;
  uint8_t *s;
  __host__ __device__ __forceinline__ uint32_t get(int p) const { return s[p & (kPair - 1)]; }
  __host__ __device__ __forceinline__ void set(int p, uint32_t v) const {
    w.sync();
    s[p & (kPair - 1)] = static_cast<uint8_t>(v);
  }
};
template <class Tape>
__host__ __device__ __forceinline__ void reset_tape(const Tape t, int pos) {
  forth_reset(t, pos);
}
template <class W>
__host__ __device__ __forceinline__ void reset_tape(const TrackedBytes<W> t, int pos) {
  const uint64_t seed = reset_seed(t.s);
  t.w.sync();
  t.w.each([&](uint32_t l) {
    for (uint32_t i = l; i < kTape; i += kWarp) t.s[i] = reset_byte(seed, pos, i);
  });
  t.w.sync();
  t.written.lo0 = 0;
  t.written.hi0 = kTape - 1;
}

// Where a program stands.  The top two stack entries live in registers (r0 =
// stack[sp - 1], r1 = stack[sp - 2]); memory holds stack[0 .. sp - 2).  Most
// ops then touch no memory for their stack traffic: a push spills the entry it
// pushes down, a pop refills the second entry, neither on the step's own
// dependency chain.  Stack slots at or above sp hold anything; they are never
// read before a push overwrites them.
struct ForthState {
  int pos, sp;
  bool overflow;
  uint32_t r0, r1;         // stack[sp - 1], stack[sp - 2] (when they exist)
  uint32_t i, nops, mods;  // raw steps, no-ops, value-changing tape writes

  __host__ __device__ __forceinline__ void begin() {
    pos = sp = 0;
    overflow = false;
    r0 = r1 = 0;
    i = nops = mods = 0;
  }
};

template <bool kWithReset>
struct ForthLane {
  ForthState st;

  template <class Tape>
  __host__ __device__ __forceinline__ void push(const Tape stk, uint32_t v) {
    if (st.sp != kPair) {
      if (st.sp >= 2) stk.set(st.sp - 2, st.r1);
      st.r1 = st.r0;
      st.r0 = v & 0xFF;
      st.sp++;
    } else {
      st.overflow = true;
    }
  }

  template <class Tape>
  __host__ __device__ __forceinline__ uint32_t pop(const Tape stk) {
    if (st.sp == 0) return 0u;
    const uint32_t v = st.r0;
    st.sp--;
    st.r0 = st.r1;
    if (st.sp >= 2) st.r1 = stk.get(st.sp - 2);
    return v;
  }
  template <class Tape>
  __host__ __device__ __forceinline__ void write(const Tape t, int a, uint32_t v) {
    v &= 0xFF;
    if (t.get(a) != v) {
      t.set(a, v);
      st.mods++;
    }
  }

  // The step at st.pos, whose byte is c, of op `op` (back: it jumped
  // backwards); returns true when the program has ended.
  template <class Tape, class Stack>
  __host__ __device__ __forceinline__ bool execute(const Tape t, const Stack stk, uint32_t op,
                                                   uint32_t c, bool &back) {
    back = false;
    switch (op) {
      case kRead0: { const int a = pop(stk) % kTape; push(stk, t.get(a)); break; }
      case kRead1: { const int a = pop(stk) % kTape; push(stk, t.get(kTape + a)); break; }
      case kRead: { const int a = pop(stk) % kPair; push(stk, t.get(a)); break; }
      case kWrite: {
        const uint32_t v = pop(stk);
        const int a = pop(stk) % kPair;
        write(t, a, v);
        break;
      }
      case kWrite0: {
        const uint32_t v = pop(stk);
        const int a = pop(stk) % kTape;
        write(t, a, v);
        break;
      }
      case kWrite1: {
        const uint32_t v = pop(stk);
        const int a = pop(stk) % kTape;
        if (kWithReset && t.get(kTape + a) == 0x13) {
          reset_tape(t, st.pos);
          st.mods++;
        } else {
          write(t, kTape + a, v);
        }
        break;
      }
      case kDup: { const uint32_t v = pop(stk); push(stk, v); push(stk, v); break; }
      case kDrop: pop(stk); break;
      case kSwap: {
        const uint32_t a = pop(stk), b = pop(stk);
        push(stk, a);
        push(stk, b);
        break;
      }
      case kIf0: {
        const uint32_t v = pop(stk);
        if (v) st.pos++;
        push(stk, v);
        break;
      }
      case kInc: push(stk, pop(stk) + 1); break;
      case kDec: push(stk, pop(stk) - 1); break;
      case kAdd: { const uint32_t a = pop(stk), b = pop(stk); push(stk, a + b); break; }
      case kSub: { const uint32_t a = pop(stk), b = pop(stk); push(stk, a - b); break; }
      case kConst: push(stk, c & 63); break;
      case kCopy0: {
        const int a = pop(stk) % kTape;
        if (kWithReset && t.get(kTape + a) == 0x13) {
          reset_tape(t, st.pos);
          st.mods++;
        } else {
          write(t, kTape + a, t.get(a));
        }
        break;
      }
      case kCopy1: { const int a = pop(stk) % kTape; write(t, a, t.get(kTape + a)); break; }
      case kCopy: {
        const int to = pop(stk) % kPair;
        const int from = pop(stk) % kPair;
        write(t, to, t.get(from));
        break;
      }
      case kXor: push(stk, pop(stk) ^ 64); break;
      case kJmp: {
        const int a = (c & 63) + 1;
        st.pos += (c & 64) ? -a : a;
        st.pos--;
        back = (c & 64) != 0;
        break;
      }
      default: st.nops++;
    }
    st.pos++;
    st.i++;
    if (st.pos >= kPair || st.pos < 0 || st.overflow || st.i >= kStepLimit) return true;
    return false;
  }
  template <class Tape, class Stack>
  __host__ __device__ __forceinline__ bool step(const Tape t, const Stack stk,
                                                const uint8_t *__restrict__ optab, bool &back) {
    const uint32_t c = t.get(st.pos);
    return execute(t, stk, optab[c], c, back);
  }
};

// What a lane's cycle check keeps of a program.
struct ForthCycle {
  int pos, sp;  // of the snapshot (pos -1: none)
  uint32_t i, nops, mods, top, power, lam;
  uint64_t mem;
};

// The first steps of a program on one lane; and any number more (step_on), with
// exact cycle fast-forward at backward jumps on Brent's schedule (cycle.cuh), for
// stacks of up to 8 entries, compared byte by byte, and an unchanged tape.
template <bool kWithReset>
struct ForthFirst {
  using Cycle = ForthCycle;
  // Most random programs end within 24 steps (90 % of those of a soup of 2^15
  // forth programs after 256 epochs).
  static constexpr uint32_t kSteps = 24;
  enum Status : uint32_t { kRuns, kEnds, kJumps };
  ForthLane<kWithReset> ln;
  uint32_t status;

  template <class Tape>
  __host__ __device__ __forceinline__ void begin(const Tape, Mask128, const uint8_t *) {
    ln.st.begin();
    status = kRuns;
  }
  template <class Tape>
  __host__ __device__ __forceinline__ void step(const Tape t, const Tape stk,
                                                const uint8_t *__restrict__ optab) {
    bool back;
    status = ln.step(t, stk, optab, back) ? kEnds : ln.st.i >= kSteps ? kJumps : kRuns;
  }
  template <class Tape>
  __host__ __device__ __forceinline__ void resolve(const Tape, const uint8_t *) {}

  __host__ __device__ __forceinline__ static void begin_cycle(ForthCycle &y) {
    y.pos = -1;
    y.power = 1;
    y.lam = 0;
  }
  // A step of a program that goes on (kJumps); kEnds when it was the last.
  template <class Tape>
  __host__ __device__ __forceinline__ void step_on(const Tape t, const Tape stk,
                                                   const uint8_t *__restrict__ optab,
                                                   ForthCycle &y) {
    bool back;
    bool ends = ln.step(t, stk, optab, back);
    if (!ends && back) {
      visit(stk, y);
      ends = ln.st.i >= kStepLimit;
    }
    if (ends) status = kEnds;
  }
  template <class Tape>
  __host__ __device__ __forceinline__ void settle(const Tape, const Tape, const uint8_t *) {}
  // stack[0 .. sp - 2), the entries below the registers, packed.
  template <class Tape>
  __host__ __device__ __forceinline__ uint64_t below(const Tape stk) const {
    uint64_t w = 0;
    for (int j = 0; j < ln.st.sp - 2; j++) w |= static_cast<uint64_t>(stk.get(j)) << (8 * j);
    return w;
  }
  template <class Tape>
  __host__ __device__ __forceinline__ void visit(const Tape stk, ForthCycle &y) {
    ForthState &st = ln.st;
    const uint32_t top = (st.sp >= 1 ? st.r0 : 0u) | (st.sp >= 2 ? st.r1 : 0u) << 8;
    if (st.pos == y.pos && top == y.top && st.sp == y.sp && st.mods == y.mods &&
        (st.sp <= 2 || below(stk) == y.mem)) {
      const uint32_t len = st.i - y.i, k = (kStepLimit - st.i) / len;
      st.i += k * len;
      st.nops += k * (st.nops - y.nops);
    }
    if (++y.lam == y.power) {
      y.pos = st.sp <= 8 ? st.pos : -1;  // larger stacks: no snapshot
      y.sp = st.sp;
      y.mods = st.mods;
      y.i = st.i;
      y.nops = st.nops;
      y.top = top;
      y.mem = st.sp > 2 && st.sp <= 8 ? below(stk) : 0;
      y.power <<= 1;
      y.lam = 0;
    }
  }
  __host__ __device__ __forceinline__ const ForthState &state() const { return ln.st; }
  __host__ __device__ __forceinline__ uint32_t ops() const { return ln.st.i - ln.st.nops; }
  __host__ __device__ __forceinline__ uint32_t raw() const { return ln.st.i; }
  __host__ __device__ __forceinline__ uint32_t mods() const { return ln.st.mods; }
};

// Shared memory of one warp's ForthWarp.
struct alignas(16) ForthMem {
  uint8_t T[kPair];      // the pair tape
  uint8_t stk[kPair];    // the stack
  uint8_t snap[kPair];   // their snapshots
  uint8_t ssnap[kPair];
  uint32_t E[kPair];     // where a run of jumps and no-ops leads (ForthWarp)
  uint16_t R[kPair];     // lowest | highest << 8 of the positions it depends on
};

// One pair on a whole warp.
//
// What bounds it: the chain of dependent instructions of one program (~5
// cycles each), and most steps of the programs that run long are jumps (44 %)
// and no-ops (22 %), which change nothing but the position.  So all 128
// positions are decoded at once into where the run of jumps and no-ops from
// there leads: E[p] = q | steps << 8 | no-ops << 16 | code << 24, with q the
// first position that holds another op (code: the op, or kConstant | value) or
// kPair where the run leaves the tape.  The lanes find it by pointer doubling:
// a run of up to 2^r steps is resolved after r rounds, and one not resolved
// after 7 goes in circles (its entry then leads 128 steps ahead).  Writes only
// widen the ranges of positions changed since; an entry is used when no
// position it depends on (R) lies in them, else all are decoded again; a
// program that changes its own code all the time is stepped through plainly.
//
// Exact cycle fast-forward where a run leads backwards, on Brent's schedule
// (cycle.cuh): the state is (position, stack, tape); the two registers are
// compared first, then stack and tape with their snapshots, four bytes per
// lane.  Less will do for a segment without an if0 or a tape write ("blind"):
// nothing it does depends on a value but other values, so back at the same
// position and depth it repeats to the step limit whatever is on the stack;
// and one that leaves the stack deeper by d without having met its bottom
// repeats, d deeper each time, until the stack overflows.
//
// Stores to the tape and the stack are made by every lane alike, each after a
// sync (as in BffWarp): by then all lanes have read what it changes and made the
// store before it.
template <class W, bool kWithReset>
struct ForthWarp {
  static constexpr uint32_t kConstant = 64, kOut = 62, kPending = 63;  // codes
  static constexpr uint32_t kPlainSteps = 64;

  const W w;
  ForthMem &m;
  const uint8_t *const optab;
  ForthLane<kWithReset> ln;
  Written written;       // since the decode
  uint32_t since;        // ops executed since the decode
  // Snapshot.
  int s_key, s_sp;
  uint32_t s_r0, s_r1, s_i, s_nops, s_mods, s_power, s_lam;
  // Since the snapshot: no if0 or tape write; a pop found the stack empty; the
  // deepest stack.
  bool blind, bottom;
  int deepest;

  __host__ __device__ __forceinline__ ForthWarp(W warp, ForthMem &mem, const uint8_t *table)
      : w(warp), m(mem), optab(table) {}

  __host__ __device__ __forceinline__ uint32_t word(const uint8_t *a, uint32_t l) const {
    return reinterpret_cast<const uint32_t *>(a)[l];
  }

  __host__ __device__ __forceinline__ void decode() {
    written.clear();
    since = 0;
    w.sync();
    w.each([&](uint32_t l) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int p = static_cast<int>(32 * k + l);
        const uint32_t b = m.T[p], op = optab[b];
        int q = p;
        uint32_t e = (op == kConst ? kConstant | (b & 63) : op) << 24;
        if (op == kFNoop || op == kJmp) {
          const int a = static_cast<int>(b & 63) + 1;
          q = op == kFNoop ? p + 1 : (b & 64) ? p - a : p + a;
          const bool out = q < 0 || q >= kPair;
          e = (out ? kOut : kPending) << 24 | (op == kFNoop ? 1u << 16 : 0u) | 1u << 8;
          if (out) q = kPair;
        }
        m.E[p] = e | static_cast<uint32_t>(q);
        m.R[p] = static_cast<uint16_t>(p | p << 8);
      }
    });
    w.sync();
    for (int round = 0; round < 7; round++) {
      struct Entries {
        uint32_t e[4], r[4];
      };
      const auto next = w.map([&](uint32_t l) {
        Entries x;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t e = m.E[32 * k + l], r = m.R[32 * k + l];
          x.e[k] = e;
          x.r[k] = r;
          if ((e >> 24) == kPending) {
            const uint32_t f = m.E[e & 0xFF], g = m.R[e & 0xFF];
            x.e[k] = f + (e & 0x00FFFF00u);
            const uint32_t lo = (r & 0xFF) < (g & 0xFF) ? r & 0xFF : g & 0xFF;
            const uint32_t hi = (r >> 8) > (g >> 8) ? r >> 8 : g >> 8;
            x.r[k] = lo | hi << 8;
          }
        }
        return x;
      });
      w.sync();
      const bool more = w.any([&](uint32_t l) {
        bool pending = false;
        const Entries x = next(l);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          m.E[32 * k + l] = x.e[k];
          m.R[32 * k + l] = static_cast<uint16_t>(x.r[k]);
          pending |= (x.e[k] >> 24) == kPending;
        }
        return pending;
      });
      w.sync();
      if (!more) break;
    }
  }

  // At position `key`, which a run led back to.
  __host__ __device__ __forceinline__ void visit(int key) {
    ForthState &st = ln.st;
    if (key == s_key && st.i < kStepLimit) {
      const int deeper = st.sp - s_sp;
      uint32_t most = 0;  // segments that may be skipped
      if (blind) {
        if (deeper == 0) most = kStepLimit;
        else if (deeper > 0 && !bottom && st.sp + deepest - s_sp + deeper <= kPair)
          most = static_cast<uint32_t>((kPair - (deepest - s_sp) - st.sp) / deeper);
      } else if (deeper == 0 && (st.sp < 1 || st.r0 == s_r0) && (st.sp < 2 || st.r1 == s_r1)) {
        const bool differs = w.any([&](uint32_t l) {
          const int b = st.sp - 2 - 4 * static_cast<int>(l);  // entries in memory
          const uint32_t use = b >= 4 ? ~0u : b <= 0 ? 0u : ~0u >> (32 - 8 * b);
          return ((word(m.stk, l) ^ word(m.ssnap, l)) & use) != 0 ||
                 (st.mods != s_mods && word(m.T, l) != word(m.snap, l));
        });
        if (!differs) most = kStepLimit;
      }
      if (most != 0) {
        const uint32_t len = st.i - s_i, room = (kStepLimit - st.i) / len;
        const uint32_t k = most < room ? most : room;
        st.i += k * len;
        st.nops += k * (st.nops - s_nops);
        st.sp += static_cast<int>(k) * deeper;
        deepest += static_cast<int>(k) * deeper;
      }
    }
    if (++s_lam == s_power) {
      s_key = key;
      s_sp = st.sp;
      s_r0 = st.r0;
      s_r1 = st.r1;
      s_i = st.i;
      s_nops = st.nops;
      s_mods = st.mods;
      s_power <<= 1;
      s_lam = 0;
      blind = true;
      bottom = false;
      deepest = st.sp;
      w.each([&](uint32_t l) {
        reinterpret_cast<uint32_t *>(m.snap)[l] = word(m.T, l);
        reinterpret_cast<uint32_t *>(m.ssnap)[l] = word(m.stk, l);
      });
    }
  }

  // The jumps and no-ops from position p up to the step limit, which comes
  // before anything else.
  __host__ __device__ __forceinline__ void run_out(int p) {
    ForthState &st = ln.st;
    while (st.i < kStepLimit) {
      const uint32_t b = m.T[p & (kPair - 1)];
      if (optab[b] == kFNoop) {
        st.nops++;
        p++;
      } else {
        p += (b & 64) ? -static_cast<int>(b & 63) - 1 : static_cast<int>(b & 63) + 1;
      }
      st.i++;
    }
  }

  // Writes v at position a.
  __host__ __device__ __forceinline__ void write(int a, uint32_t v) {
    blind = false;
    if (m.T[a] != v) {
      w.sync();
      m.T[a] = static_cast<uint8_t>(v);
      ln.st.mods++;
      written.add(a);
    }
  }
  // The second register after a pop.
  __host__ __device__ __forceinline__ void refill() {
    if (ln.st.sp >= 2) ln.st.r1 = m.stk[ln.st.sp - 2];
  }
  __host__ __device__ __forceinline__ void drop() {
    ForthState &st = ln.st;
    bottom |= st.sp == 0;
    if (st.sp == 0) return;
    st.sp--;
    st.r0 = st.r1;
    refill();
  }
  __host__ __device__ __forceinline__ void push(uint32_t v) {
    ForthState &st = ln.st;
    if (st.sp == kPair) {
      st.overflow = true;
      return;
    }
    if (st.sp >= 2) {
      w.sync();
      m.stk[st.sp - 2] = static_cast<uint8_t>(st.r1);
    }
    st.r1 = st.r0;
    st.r0 = v;
    st.sp++;
    deepest = st.sp > deepest ? st.sp : deepest;
  }
  // The top entry, 0 when there is none, which it then becomes.
  __host__ __device__ __forceinline__ uint32_t top() {
    ForthState &st = ln.st;
    if (st.sp == 0) {
      bottom = true;
      st.sp = 1;
      st.r0 = 0;
    }
    return st.r0;
  }
  // Pops two entries: v on top of a.
  __host__ __device__ __forceinline__ void pop2(uint32_t &v, uint32_t &a) {
    ForthState &st = ln.st;
    bottom |= st.sp < 2;
    v = st.sp >= 1 ? st.r0 : 0u;
    a = st.sp >= 2 ? st.r1 : 0u;
    if (st.sp >= 3) st.r0 = m.stk[st.sp - 3];
    st.sp = st.sp >= 2 ? st.sp - 2 : 0;
    refill();
  }

  // The op `code` at st.pos, as ForthLane::execute.
  __host__ __device__ __forceinline__ void operate(uint32_t code) {
    ForthState &st = ln.st;
    st.pos++;
    st.i++;
    if (code >= kConstant) {
      push(code & 63);
      return;
    }
    switch (code) {
      case kInc: st.r0 = (top() + 1) & 0xFF; break;
      case kDec: st.r0 = (top() - 1) & 0xFF; break;
      case kXor: st.r0 = top() ^ 64; break;
      case kRead0: st.r0 = m.T[top() % kTape]; break;
      case kRead1: st.r0 = m.T[kTape + top() % kTape]; break;
      case kRead: st.r0 = m.T[top() % kPair]; break;
      case kIf0:
        blind = false;
        st.pos += top() != 0;
        break;
      case kDrop: drop(); break;
      case kDup: {
        const uint32_t v = top();
        push(v);
        break;
      }
      case kAdd:
      case kSub: {
        const uint32_t a = top(), b = st.sp >= 2 ? st.r1 : 0u;
        bottom |= st.sp < 2;
        if (st.sp >= 2) {
          st.sp--;
          refill();
        }
        st.r0 = (code == kAdd ? a + b : a - b) & 0xFF;
        break;
      }
      case kSwap: {
        const uint32_t a = top();
        st.r0 = st.sp >= 2 ? st.r1 : 0u;
        st.r1 = a;
        bottom |= st.sp < 2;
        if (st.sp < 2) st.sp = 2;
        break;
      }
      case kWrite0:
      case kWrite1:
      case kWrite: {
        uint32_t v, a;
        pop2(v, a);
        const int p = code == kWrite ? a % kPair : code == kWrite1 ? kTape + a % kTape : a % kTape;
        if (kWithReset && code == kWrite1 && m.T[p] == 0x13) reset();
        else write(p, v);
        break;
      }
      case kCopy: {
        uint32_t to, from;
        pop2(to, from);
        write(to % kPair, m.T[from % kPair]);
        break;
      }
      default: {  // kCopy0, kCopy1
        const int a = (st.sp >= 1 ? st.r0 : 0u) % kTape;
        drop();
        const int to = code == kCopy0 ? kTape + a : a;
        if (kWithReset && code == kCopy0 && m.T[to] == 0x13) reset();
        else write(to, m.T[to ^ kTape]);
        break;
      }
    }
  }
  __host__ __device__ __forceinline__ void reset() {
    reset_tape(TrackedBytes<W>{w, m.T, written}, ln.st.pos - 1);
    ln.st.mods++;
    blind = false;
  }

  // The state at the start of a program.
  __host__ __device__ __forceinline__ ForthState start(bool) const {
    ForthState s;
    s.begin();
    return s;
  }

  // Runs the program in m.T, with the stack in m.stk, from state s to its end.
  __host__ __device__ __forceinline__ void run(const ForthState &s) {
    ln.st = s;
    ForthState &st = ln.st;
    s_key = -1;
    s_sp = 0;
    s_r0 = s_r1 = s_i = s_nops = s_mods = s_lam = 0;
    s_power = 1;
    blind = bottom = false;
    deepest = 0;
    decode();
    uint32_t plain = 0;  // steps to take one by one
    int last = -1;
    while (true) {
      if (plain != 0) {
        const TrackedBytes<W> t{w, m.T, written};
        bool back;
        blind = false;  // (not tracked here)
        if (ln.step(t, StackBytes<W>{w, m.stk}, optab, back)) return;
        if (back) {
          visit(st.pos);
          if (st.i >= kStepLimit) return;
        }
        if (--plain == 0) {
          decode();
          last = -1;  // (the last step's visit, if any, was for this very state)
        }
        continue;
      }
      const uint32_t e = m.E[st.pos], r = m.R[st.pos];
      if (!written.none() && written.meets(static_cast<int>(r & 0xFF), static_cast<int>(r >> 8))) {
        if (since < 8) plain = kPlainSteps;
        else decode();
        continue;
      }
      const uint32_t steps = (e >> 8) & 0xFF, code = e >> 24;
      if (st.i + steps >= kStepLimit) {
        run_out(st.pos);
        return;
      }
      st.i += steps;
      st.nops += (e >> 16) & 0xFF;
      st.pos = static_cast<int>(e & 0xFF);
      if (code == kOut) return;
      if (code == kPending) continue;  // in circles, 128 steps at a time
      if (st.pos <= last) {
        visit(st.pos);
        if (st.i >= kStepLimit) return;
      }
      last = st.pos;
      since++;
      operate(code);
      if (st.pos >= kPair || st.overflow || st.i >= kStepLimit) return;
    }
  }

  __host__ __device__ __forceinline__ uint32_t ops() const { return ln.st.i - ln.st.nops; }
  __host__ __device__ __forceinline__ uint32_t raw() const { return ln.st.i; }
  __host__ __device__ __forceinline__ uint32_t mods() const { return ln.st.mods; }
};

}  // namespace cubff

// pipeline_kernel.cuh — the kernel that runs epochs of one or more soups as one
// dataflow pipeline instead of one launch per epoch.
//
// Pair k of epoch e reads programs s_e[2k], s_e[2k+1] as epoch e-1 left them
// and writes them back; nothing else of epoch e-1 matters to it.  So a pair
// may start as soon as the two pairs of epoch e-1 that wrote its programs are
// done, while long-running pairs elsewhere are still being interpreted: the
// 8192-step tail of an epoch only delays its own dependency cone.  Soups are
// independent, so a batch of soups of one language (any sizes and mutation
// rates) shares one persistent launch and one ready queue.
//
// Every wait is bounded (10 s of %globaltimer by default); a timeout sets
// *error = 1, the waiting lanes give up, and the host reports CUBFF_ETIMEDOUT.
// A ready-queue entry naming no task of the launch sets *error = 2 (reported
// as CUBFF_EDEVICE) instead of being used as an index.  Results are
// bit-identical to the per-epoch launches: every program sees the same
// sequence of pair operations (MutateAndRunPrograms, common_language.h:163-192)
// with the same inputs.
#pragma once

#include "epoch_body.cuh"
#include "launch_plan.h"
#include "staged.cuh"

namespace cubff {
namespace {

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void fence_acq_rel_gpu() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kCountSlots = kPipeCountSlots;  // per-epoch counter slots (spread the atomics)

// Ready-queue dataflow over one or more soups.  A pair of epoch e+1 can run
// once the two pairs of epoch e that wrote its programs are done.  A finished
// pair notifies the consumers of its two programs (inv gives a program's
// position in the next epoch's shuffle, hence its pair); the second
// notification of a consumer pushes it into its language's ready queue.
// Epoch-0 pairs of the launch are implicitly ready (the first `initial`
// slots of each queue).  Warps claim queue slots in bulk, so the lanes they
// hand out stage their pairs together.  Every pushed task is runnable, so no
// lane ever waits on a dependency; a lane only waits for a claimed slot to be
// written, and every slot below a queue's task count is eventually written
// (all pairs of epoch e complete => all of epoch e+1 are pushed).
//
// A launch serves the soups of one language through one queue (the soups of
// other languages run in launches of their own, on other streams).
//
// No global access is consumed in the iteration that issues it where that
// can be avoided: queue entries and shuffle indices land in registers read
// back in a later iteration.  Lane states:
//   idle -> slot (wait for the entry) -> index -> run [-> long] -> notify -> idle
// and `exhausted` once a claim falls past the queue's last task.
//
// How a warp runs its pairs depends on the language family (LaneServer,
// StagedServer), how many it holds at once on the size of the launch (launch_plan.h).
// Launch-shape knobs (PipeTuning, chosen by the host; the BFF and Forth families run
// a pair to its end and use none of them):
//  * steps_per_visit: interpreter steps a running lane takes per iteration of
//    its warp after its first (an iteration lasts as long as its busiest
//    lane, so a lane given more steps holds its warp-mates, and the pairs
//    they would finish and notify, for its extra steps);
//  * first_visit_steps: the steps of a pair's first visit.  Lanes that claim
//    together stage and start together, and most pairs end within a few
//    steps; the first visit's budget bounds how long one heavy pair among
//    them holds the others (whose consumers wait on them) before they can
//    write back;
//  * claim_min: a warp with running lanes claims new slots only once this
//    many of 32 of its lanes, in proportion, are idle (an idle warp claims at once;
//    at 32, the default, no other does), so a slot held by a busy warp is polled
//    only between its long iterations;
//  * long_visits: a pair still running after this many visits is long.  A
//    warp holding a long pair claims nothing new: its other lanes drain, and
//    the long pair, which the next epochs' pairs wait on, steps without
//    warp-mates whose staging and steps would interleave with its own.  Few
//    pairs are long (a random 2^17-program soup has ~10-25 pairs per epoch
//    past 64 steps, out of 65536), so little capacity is set aside.

__device__ __forceinline__ uint32_t atom_add_relaxed(uint32_t *p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

__device__ __forceinline__ void st_release_u32(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

enum : uint32_t { kIdle, kSlot, kIndex, kRun, kLong, kNotify, kExhausted };

// Per-lane state of a held queue slot and its pair.
struct Lane {
  uint32_t state, slot, task, e, k, p1, p2, qv, poll_in, err, j1, j2, c1, c2;
  int si;  // soup index of the task
  uint64_t qp, t_wait;
  bool dirty, evaluated, has_next;

  __device__ __forceinline__ void begin() {
    state = kIdle;
    slot = task = e = k = p1 = p2 = qv = 0;
    poll_in = err = j1 = j2 = c1 = c2 = 0;
    si = 0;
    qp = t_wait = 0;
    dirty = evaluated = has_next = false;
  }
};

// What a warp needs of the launch: the soup descriptors (in shared memory)
// and the error flag.
struct PipeCtx {
  const PipeSoup *soups;
  int *error;
  uint64_t wait_limit_ns;
  PipeTuning tune;
};

// Soup of global task `task` among soups [lo, hi) (sorted by task_base).
__device__ __forceinline__ int soup_of_task(const PipeSoup *soups, int lo, int hi, uint32_t task) {
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (soups[mid].task_base <= task) lo = mid; else hi = mid;
  }
  return lo;
}

// Soup of epoch-0 slot `slot` among soups [lo, hi) (sorted by init_base).
__device__ __forceinline__ int soup_of_slot(const PipeSoup *soups, int lo, int hi, uint32_t slot) {
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (soups[mid].init_base <= slot) lo = mid; else hi = mid;
  }
  return lo;
}

// Claims the next queue slots for the lanes of mask `idle` (warp-uniform,
// non-zero).
__device__ __forceinline__ void claim(const PipeCtx &b, const PipeQueue &q, Lane &ln,
                                      uint32_t idle, uint32_t lane) {
  const uint32_t lt_mask = (1u << lane) - 1;
  const int s_lo = static_cast<int>(q.first_soup), s_hi = static_cast<int>(q.first_soup + q.n_soups);
  const int leader = __ffs(idle) - 1;
  uint32_t base = 0;
  if (lane == static_cast<uint32_t>(leader)) base = atomicAdd(q.ctl, __popc(idle));
  base = __shfl_sync(0xffffffffu, base, leader);
  if ((idle >> lane) & 1) {
    ln.slot = base + __popc(idle & lt_mask);
    if (ln.slot >= q.total) {
      ln.state = kExhausted;
    } else if (ln.slot < q.initial) {  // a first-epoch pair: ready
      ln.si = soup_of_slot(b.soups, s_lo, s_hi, ln.slot);
      const PipeSoup &sp = b.soups[ln.si];
      ln.task = sp.task_base + (ln.slot - sp.init_base);
      ln.state = kIndex;
      ln.qp = *reinterpret_cast<const unsigned long long *>(sp.perm + 2 * uint64_t(ln.slot - sp.init_base));
    } else {
      ln.state = kSlot;
      ln.qv = ld_relaxed(q.queue + (ln.slot - q.initial));
      ln.poll_in = 0;
      ln.t_wait = 0;
    }
  }
}

// A lane in kSlot: its slot's entry, loaded in an earlier iteration, is taken
// up or loaded again.  Returns true when it was there.  Every other iteration
// loads: a consumer starts that much sooner than with a gap that grows to 16
// (64 epochs of 1022 bff_noheads programs: 2.04 ms, 2.22 before; a random soup
// of 2^15 bff: 5.42, 5.61); loading in each iteration costs the random soup of
// 2^17 5 % and gains nothing elsewhere.
__device__ __forceinline__ bool poll_slot(const PipeCtx &b, const PipeQueue &q, Lane &ln) {
  const int s_lo = static_cast<int>(q.first_soup), s_hi = static_cast<int>(q.first_soup + q.n_soups);
  bool progressed = false;
  if (ln.qv != 0 && ln.qv - 1 >= q.total) {
    // Only pushes of tasks of this launch fill the queue; any other value
    // is reported (error 2) instead of being used as an index.
    atomicExch(b.error, 2);
    ln.state = kExhausted;
  } else if (ln.qv != 0) {
    ln.task = ln.qv - 1;
    // Consumed: leave the entry zero for the next launch.
    q.queue[ln.slot - q.initial] = 0;
    ln.si = soup_of_task(b.soups, s_lo, s_hi, ln.task);
    const PipeSoup &sp = b.soups[ln.si];
    const uint32_t rel = ln.task - sp.task_base;
    ln.e = rel / sp.npairs;
    ln.k = rel - ln.e * sp.npairs;
    ln.qp = *reinterpret_cast<const unsigned long long *>(sp.perm + uint64_t(ln.e) * sp.n +
                                                          2 * uint64_t(ln.k));
    ln.state = kIndex;
    progressed = true;
  } else if (ln.poll_in-- == 0) {
    if (ln.err) {
      ln.state = kExhausted;
    } else {
      const uint64_t now = globaltimer_ns();
      if (ln.t_wait == 0) {
        ln.t_wait = now;
      } else if (now - ln.t_wait > b.wait_limit_ns) {
        atomicExch(b.error, 1);
        ln.state = kExhausted;
      }
    }
    if (ln.state == kSlot) {
      ln.qv = ld_relaxed(q.queue + (ln.slot - q.initial));
      ln.err = ld_relaxed(reinterpret_cast<const uint32_t *>(b.error));
      ln.poll_in = 1;
    }
  }
  return progressed;
}

// A lane in kIndex: its shuffle indices have landed.  Orders its reads after
// the producers' writes and loads the next epoch's positions of both programs.
__device__ __forceinline__ void take_index(const PipeSoup &sp, const PipeQueue &q, Lane &ln) {
  if (ln.slot < q.initial) {
    ln.e = 0;
    ln.k = ln.slot - sp.init_base;
  }
  ln.p1 = static_cast<uint32_t>(ln.qp);
  ln.p2 = static_cast<uint32_t>(ln.qp >> 32);
  fence_acq_rel_gpu();
  // Both inputs have been counted: leave the counter zero for the next launch.
  if (ln.e > 0) sp.readycnt[uint64_t(ln.e) * sp.npairs + ln.k] = 0;
  ln.has_next = ln.e + 1 < sp.n_epochs;
  if (ln.has_next) {
    ln.j1 = __ldg(sp.inv + uint64_t(ln.e + 1) * sp.n + ln.p1);
    ln.j2 = __ldg(sp.inv + uint64_t(ln.e + 1) * sp.n + ln.p2);
  }
}

// The mutations of a pair (common_language.h:172-180), whose positions mm
// marks: set(i, byte) for each.
template <class F>
__device__ __forceinline__ void mutate_bits(const PipeSoup &sp, const Lane &ln, uint4 mm, F set) {
  const uint64_t key0 = (sp.n * seed_from(sp.s0, sp.e0 + ln.e) + ln.k) * kPair;
  const uint32_t mw[4] = {mm.x, mm.y, mm.z, mm.w};
#pragma unroll
  for (int qd = 0; qd < 4; qd++) {
    uint32_t bits = mw[qd];
    while (bits) {
      const int i = qd * 32 + __ffs(bits) - 1;
      bits &= bits - 1;
      set(i, static_cast<uint32_t>(splitmix64(key0 + i)) & 0xFFu);
    }
  }
}

// Writes back the 32 words of a lane's pair: first half, then second half
// (common_language.h:188-191).
template <class F>
__device__ __forceinline__ void store_pair(const PipeSoup &sp, const Lane &ln, F word) {
  uint4 *o1 = reinterpret_cast<uint4 *>(sp.soup + uint64_t(ln.p1) * kTape);
  uint4 *o2 = reinterpret_cast<uint4 *>(sp.soup + uint64_t(ln.p2) * kTape);
#pragma unroll
  for (int qd = 0; qd < 4; qd++)
    o1[qd] = make_uint4(word(4 * qd), word(4 * qd + 1), word(4 * qd + 2), word(4 * qd + 3));
#pragma unroll
  for (int qd = 0; qd < 4; qd++)
    o2[qd] = make_uint4(word(16 + 4 * qd), word(17 + 4 * qd), word(18 + 4 * qd),
                        word(19 + 4 * qd));
}

__device__ __forceinline__ void add_counts(const PipeSoup &sp, uint32_t e, uint32_t slot_ctr,
                                           uint32_t ops, uint32_t raw) {
  unsigned long long *c = sp.ops + (uint64_t(e) * kCountSlots + slot_ctr) * 2;
  if (ops) atomicAdd(c, static_cast<unsigned long long>(ops));
  if (raw) atomicAdd(c + 1, static_cast<unsigned long long>(raw));
}

// A finished pair whose bytes have been written: notifies the consumers of its
// two programs.
__device__ __forceinline__ void finish(const PipeSoup &sp, Lane &ln) {
  if (ln.has_next) {
    // The fences order the stores before the increments, and make the earlier
    // producer's stores visible to whoever pushes; between them both increments
    // are under way together.
    uint32_t *rc = sp.readycnt + uint64_t(ln.e + 1) * sp.npairs;
    fence_acq_rel_gpu();
    ln.c1 = atom_add_relaxed(rc + (ln.j1 >> 1), 1);
    ln.c2 = atom_add_relaxed(rc + (ln.j2 >> 1), 1);
    fence_acq_rel_gpu();
    ln.state = kNotify;
  } else {
    ln.state = kIdle;
  }
}

// Pushes the consumers whose second input was a pair of a lane in kNotify.
__device__ __forceinline__ void push_ready(const PipeCtx &b, const PipeQueue &q, Lane &ln,
                                           uint32_t lane) {
  const uint32_t lt_mask = (1u << lane) - 1;
  const bool same = (ln.j2 >> 1) == (ln.j1 >> 1);
  const bool push1 = ln.state == kNotify && (ln.c1 == 1 || (same && ln.c2 == 1));
  const bool push2 = ln.state == kNotify && !same && ln.c2 == 1;
  const uint32_t nmask1 = __ballot_sync(0xffffffffu, push1);
  const uint32_t nmask2 = __ballot_sync(0xffffffffu, push2);
  if (nmask1 | nmask2) {
    const int leader = __ffs(nmask1 | nmask2) - 1;
    uint32_t base = 0;
    if (lane == static_cast<uint32_t>(leader)) base = atomicAdd(q.ctl + 1, __popc(nmask1) + __popc(nmask2));
    base = __shfl_sync(0xffffffffu, base, leader);
    const PipeSoup &sp = b.soups[ln.si];
    const uint32_t next = sp.task_base + (ln.e + 1) * sp.npairs;
    if (push1) st_release_u32(q.queue + base + __popc(nmask1 & lt_mask), next + (ln.j1 >> 1) + 1);
    if (push2)
      st_release_u32(q.queue + base + __popc(nmask1) + __popc(nmask2 & lt_mask),
                     next + (ln.j2 >> 1) + 1);
  }
  if (ln.state == kNotify) ln.state = kIdle;
}

// The SUBLEQ languages: one pair per lane, staged and run for some steps in one
// iteration.  Pairs take 4 steps on average; what an epoch takes is the chain of
// its latencies (index, programs, steps, two counters, queue) and, now and then, a
// pair of thousands of steps.  64 epochs of 2^17 subleq programs 4.18 ms (5.79 with
// tapes staged byte by byte, in an iteration of its own), of 40962 rsubleq4
// programs 3.27 ms (4.27; 3.44 with 32 pairs to a warp); shared memory for those 16
// lanes alone, instead of for 32, 5 to 8 % less for subleq.
// iterate() is one iteration of the warp; it returns true if the lane made
// progress.
template <int L>
struct LaneServer {
  SubleqMachine<(L == kRsubleq4)> m;
  uint32_t visits;
  static constexpr uint32_t kWidth = 16;  // lanes that hold pairs
  using Mem = SubleqMem<kWidth>;
  static constexpr size_t kWarpBytes = sizeof(Mem);  // of shared memory
  LaneWords<kWidth> t, snap;

  __device__ __forceinline__ LaneServer(uint8_t *smem, const uint8_t *, uint32_t tid)
      : visits(0), t{smem + (tid >> 5) * kWarpBytes, tid & 31},
        snap{t.s + sizeof(Mem::tapes), tid & 31} {}

  // Stages the pair of a lane in kIndex: bytes into shared memory, mutations.
  __device__ __forceinline__ void stage(const PipeSoup &sp, Lane &ln) {
    uint32_t w[32];
    load_pair(sp.soup, ln.p1, ln.p2, w);
    const uint4 mm = __ldg(sp.mutmask + uint64_t(ln.e) * sp.npairs + ln.k);
#pragma unroll
    for (int q = 0; q < 32; q++) t.word(q) = w[q];
    ln.dirty = (mm.x | mm.y | mm.z | mm.w) != 0;
    if (ln.dirty)
      mutate_bits(sp, ln, mm, [&](int i, uint32_t v) { t.set(i, v); });
    const uint64_t num_indices = sp.num_indices ? sp.num_indices[ln.e] : sp.npairs;
    ln.evaluated = ln.k < num_indices;
    m.begin();
    visits = 0;
  }

  __device__ __forceinline__ bool iterate(const PipeCtx &b, const PipeQueue &q, Lane &ln,
                                          uint32_t lane, uint32_t slot_ctr) {
    // 1. Bulk claim of queue slots by idle lanes.
    const uint32_t idle = __ballot_sync(0xffffffffu, ln.state == kIdle);
    const uint32_t busy = __ballot_sync(0xffffffffu, ln.state != kIdle && ln.state != kExhausted);
    const uint32_t lng = __ballot_sync(0xffffffffu, ln.state == kRun && visits >= b.tune.long_visits);
    if (idle && (busy == 0 || (lng == 0 && idle_enough(__popc(idle), kWidth, b.tune.claim_min))))
      claim(b, q, ln, idle, lane);
    bool progressed = false;

    if (ln.state == kSlot) {
      // 2. Waiting for the claimed slot's entry (polled in an earlier iteration).
      progressed = poll_slot(b, q, ln);
    } else if (ln.state == kIndex) {
      // 3. Shuffle indices landed: gather and stage the pair.
      const PipeSoup &sp = b.soups[ln.si];
      take_index(sp, q, ln);
      stage(sp, ln);
      ln.state = kRun;
      progressed = true;
    }
    // 4. Some steps; pairs that ended: write back and notify.
    bool fin = false;
    if (ln.state == kRun) {
      progressed = true;
      fin = !ln.evaluated;
      const uint32_t steps = visits ? b.tune.steps_per_visit : b.tune.first_visit_steps;
      for (uint32_t r = 0; r < steps && !fin; r++) fin = m.step(t, snap);
      visits++;
      if (fin) {
        const PipeSoup &sp = b.soups[ln.si];
        if (ln.dirty || (ln.evaluated && m.mods != 0))
          store_pair(sp, ln, [&](int qd) { return t.word(qd); });
        finish(sp, ln);
      }
    }
    // The counts of the pairs that ended, summed over those of one soup and
    // epoch: pairs are so short that the atomics of each would queue up on the
    // epoch's few counters (64 epochs of 2^17 subleq programs: 4.50 ms, 5.23 with
    // them).
    for (uint32_t left = __ballot_sync(0xffffffffu, fin && ln.evaluated); left != 0;) {
      const int first = __ffs(left) - 1;
      const uint32_t e = __shfl_sync(0xffffffffu, ln.e, first);
      const int si = __shfl_sync(0xffffffffu, ln.si, first);
      const bool mine = ((left >> lane) & 1) && ln.e == e && ln.si == si;
      const uint32_t ops = __reduce_add_sync(0xffffffffu, mine ? m.ops() : 0);
      if (lane == static_cast<uint32_t>(first)) add_counts(b.soups[si], e, slot_ctr, ops, ops);
      left &= ~__ballot_sync(0xffffffffu, mine);
    }
    // 5. Push the consumers whose second input this pair was.
    push_ready(b, q, ln, lane);
    return progressed;
  }
};

// The BFF and Forth families.  The lanes of a warp run the first part of a
// pair each (BFF: up to the first jump; Forth: a few steps): most random
// programs end there, and those pairs are written back and their consumers
// notified at once.  The pairs that go on are kept (kLong) and run one after the
// other on the whole warp, one per iteration, so that slots held by other lanes are
// still polled in between.
//
// Where the warp would run such a pair command by command (Forth, and the BFF
// languages without matched brackets), and most pairs of a claim go on, as in a
// soup of self-replicators, the lanes take them on side by side instead: their
// programs are much alike, and a command of 8 costs what a command of one does.
// Once that was so, the next claim's are run so from the start, however few of
// them are there yet.  (64 epochs of forthtrivial evolved for 4096: 2^14 programs
// 82 ms, one after the other 594; bff8 2^17: 178, 340.  With 5 of 8 instead of 6
// Forth soups with some long pairs lose 5 to 15 %, as each waits for the slowest;
// with 7 instead of all of 8 bff8 soups up to 30 %, and with 20 of 32 instead of 28
// as much again.  The last eighth of a warp's pairs goes back to the whole warp in
// bff8: 2^16 evolved programs 84 ms, 104 if not; forthtrivial 2^12 would lose half.)
//
// So that pairs wait behind few others, a warp holds 8 unless there are very many
// (launch_plan.h): a soup of 2^17 bff programs taken over by self-replicators takes
// 28 ms for 16 epochs with 8 (32 lanes: about twice that), one of 1022 bff_noheads
// programs 1.8 ms for 64.
template <int L, uint32_t kLanes>
struct StagedServer {
  using LaneM = typename Stages<L>::Lane;
  using Mem = StagedMem<L, kLanes>;
  static constexpr uint32_t kWidth = kLanes;
  static constexpr size_t kWarpBytes = sizeof(Mem);
  LaneM m;
  Mem &mem;
  LaneWords<kWidth> t, stk;
  const uint8_t *optab, *cmdflag;
  static constexpr int kCrowd = Stages<L>::crowd(kLanes), kLast = Stages<L>::last(kLanes);
  static constexpr int kCrowdSteps = 256;  // of a lane in an iteration
  bool crowd;   // the lanes take pairs on themselves
  int went_on;  // pairs of this claim that went on

  __device__ __forceinline__ StagedServer(uint8_t *smem, const uint8_t *tables, uint32_t tid)
      : mem(reinterpret_cast<Mem *>(smem)[tid >> 5]), t(mem.tape(tid & 31)),
        stk(mem.stack(tid & 31)), optab(tables), cmdflag(tables + 256), crowd(false), went_on(0) {
    m.status = LaneM::kEnds;
  }

  // Some steps of a lane's long pair.  (A function of its own: inlined, what it is
  // rarely needed for slows the code around it by 4 to 8 %.)
  static __device__ __noinline__ void take_on(LaneM &pair, const LaneWords<kWidth> t,
                                              const LaneWords<kWidth> stk,
                                              const uint8_t *optab,
                                              typename LaneM::Cycle &cycle) {
    LaneM m = pair;  // (in registers)
    for (int r = 0; r < kCrowdSteps && m.status != LaneM::kEnds; r++)
      m.step_on(t, stk, optab, cycle);
    m.settle(t, stk, optab);
    pair = m;
  }

  // Stages the pair of a lane in kIndex: bytes into shared memory, command
  // mask, mutations.
  __device__ __forceinline__ void stage(const PipeSoup &sp, Lane &ln) {
    const uint4 *g1 = reinterpret_cast<const uint4 *>(sp.soup + uint64_t(ln.p1) * kTape);
    const uint4 *g2 = reinterpret_cast<const uint4 *>(sp.soup + uint64_t(ln.p2) * kTape);
    uint4 g[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      g[i] = __ldcg(g1 + i);
      g[4 + i] = __ldcg(g2 + i);
    }
    const uint4 mm = __ldg(sp.mutmask + uint64_t(ln.e) * sp.npairs + ln.k);
    Mask128 cmd{0, 0};
#pragma unroll
    for (int qd = 0; qd < 32; qd++) {
      const uint32_t w = qd % 4 == 0 ? g[qd / 4].x : qd % 4 == 1 ? g[qd / 4].y
                       : qd % 4 == 2 ? g[qd / 4].z : g[qd / 4].w;
      t.word(qd) = w;
      if (L > kBffSelfmove) continue;
      const uint32_t f = cmdflag[w & 0xFF] | (cmdflag[(w >> 8) & 0xFF] << 8) |
                         (cmdflag[(w >> 16) & 0xFF] << 16) | (cmdflag[w >> 24] << 24);
      const uint64_t nib = (f * 0x01020408u) >> 24;
      if (qd < 16) cmd.lo |= nib << (4 * qd);
      else cmd.hi |= nib << (4 * (qd - 16));
    }
    ln.dirty = (mm.x | mm.y | mm.z | mm.w) != 0;
    if (ln.dirty) {
      mutate_bits(sp, ln, mm, [&](int i, uint32_t v) {
        t.set(i, v);
        if (L <= kBffSelfmove) mask_assign(cmd, i, cmdflag[v] != 0);
      });
    }
    const uint64_t num_indices = sp.num_indices ? sp.num_indices[ln.e] : sp.npairs;
    ln.evaluated = ln.k < num_indices;
    m.begin(t, cmd, optab);
    if (!ln.evaluated) m.status = LaneM::kEnds;
  }

  // Runs the pair of lane `src` on the whole warp, writes it back and finishes
  // it.
  __device__ __forceinline__ void run_long(const PipeCtx &b, Lane &ln, uint32_t src,
                                           uint32_t lane, uint32_t slot_ctr) {
    constexpr uint32_t kAll = 0xffffffffu;
    const Counts c = run_on_warp<L>(mem.warp, mem, src, broadcast(m.state(), src), lane, optab);
    const PipeSoup &sp = b.soups[__shfl_sync(kAll, ln.si, src)];
    if (c.mods != 0 || __shfl_sync(kAll, ln.dirty, src)) {
      const uint32_t p1 = __shfl_sync(kAll, ln.p1, src), p2 = __shfl_sync(kAll, ln.p2, src);
      // First half, then second half (common_language.h:188-191): of a
      // program paired with itself the second half stays.
      if (lane >= 16 || p1 != p2)
        reinterpret_cast<uint32_t *>(sp.soup + uint64_t(lane < 16 ? p1 : p2) * kTape)[lane & 15] =
            reinterpret_cast<const uint32_t *>(mem.warp.T)[lane];
    }
    __syncwarp();  // the warp's stores before the lane's notifications
    if (lane == src) {
      if (ln.evaluated) add_counts(sp, ln.e, slot_ctr, c.ops, c.raw);
      finish(sp, ln);
    }
  }

  __device__ __forceinline__ bool iterate(const PipeCtx &b, const PipeQueue &q, Lane &ln,
                                          uint32_t lane, uint32_t slot_ctr) {
    // 1. The long pairs, or the next of them, or a bulk claim of queue slots by idle
    // lanes.
    const uint32_t lng = __ballot_sync(0xffffffffu, ln.state == kLong);
    bool together = false;
    if constexpr (Stages<L>::kCrowds) {
      crowd |= __popc(lng) >= kCrowd;
      together = crowd && __popc(lng) > kLast;
      if (together && ln.state == kLong) {
        LaneM x = m;
        take_on(x, t, stk, optab, mem.cycles[lane]);
        m = x;
        if (m.status == LaneM::kEnds) ln.state = kRun;
      }
    }
    if (!together && lng != 0) {
      run_long(b, ln, static_cast<uint32_t>(__ffs(lng) - 1), lane, slot_ctr);
    } else if (lng == 0) {
      const uint32_t idle = __ballot_sync(0xffffffffu, ln.state == kIdle);
      const uint32_t busy = __ballot_sync(0xffffffffu, ln.state != kIdle && ln.state != kExhausted);
      if (idle && busy == 0) {
        if (Stages<L>::kCrowds) {
          crowd = went_on >= kCrowd;
          went_on = 0;
        }
        claim(b, q, ln, idle, lane);
      }
    }
    bool progressed = lng != 0;

    if (ln.state == kSlot) {
      // 2. Waiting for the claimed slot's entry (polled in an earlier iteration).
      progressed |= poll_slot(b, q, ln);
    } else if (ln.state == kIndex) {
      // 3. Shuffle indices landed: gather and stage the pair.
      const PipeSoup &sp = b.soups[ln.si];
      take_index(sp, q, ln);
      stage(sp, ln);
      ln.state = kRun;
      progressed = true;
    }
    // 4. The forward parts of the pairs just staged, all lanes together.
    while (true) {
      const bool go = ln.state == kRun && m.status == LaneM::kRuns;
      if (!__any_sync(0xffffffffu, go)) break;
      if (go) m.step(t, stk, optab);
    }
    // 5. Pairs that ended: write back and notify.
    if (ln.state == kRun) {
      if (m.status == LaneM::kJumps) m.resolve(t, optab);
      if (m.status == LaneM::kJumps) {
        ln.state = kLong;
        if (Stages<L>::kCrowds) LaneM::begin_cycle(mem.cycles[lane]);
      } else {
        const PipeSoup &sp = b.soups[ln.si];
        if (ln.dirty || (ln.evaluated && m.mods() != 0))
          store_pair(sp, ln, [&](int qd) { return t.word(qd); });
        if (ln.evaluated) add_counts(sp, ln.e, slot_ctr, m.ops(), m.raw());
        finish(sp, ln);
      }
    }
    if (Stages<L>::kCrowds)
      went_on += __popc(__ballot_sync(0xffffffffu, ln.state == kLong) & ~lng);
    // 6. Push the consumers whose second input this pair was.
    push_ready(b, q, ln, lane);
    return progressed;
  }
};

template <int L, uint32_t kLanes>
using Server =
    std::conditional_t<(L <= kForthtrivialReset), StagedServer<L, kLanes>, LaneServer<L>>;

// Shared memory of a pipelined launch: the servers' (tapes and so on), the op
// and command tables, then the soup descriptors.
template <int L, uint32_t kLanes>
__host__ __device__ constexpr size_t server_bytes() {
  return (kThreads / 32) * Server<L, kLanes>::kWarpBytes;
}

// The persistent kernel of a pipelined launch over soups of language L.
// Blocks per SM set the register budget: the BFF machines take 96 without
// spills that matter (6 blocks, 80 registers: 13 % slower on the self-replicators
// above); SUBLEQ needs 76.
template <int L, uint32_t kLanes>
__global__ void __launch_bounds__(kThreads, (L <= kForthtrivialReset) ? 5 : 6)
    pipeline_kernel(const __grid_constant__ PipeBatch pb) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *tables = smem + server_bytes<L, kLanes>();
  PipeSoup *soups = reinterpret_cast<PipeSoup *>(tables + 512);
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (LangTraits<L>::kStaged) fill_tables<L>(tables);
  {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(pb.soups);
    uint32_t *dst = reinterpret_cast<uint32_t *>(soups);
    const uint32_t words = pb.n_soups * sizeof(PipeSoup) / 4;
    for (uint32_t i = tid; i < words; i += kThreads) dst[i] = src[i];
  }
  __syncthreads();  // tables and descriptors are read-only from here on
  const uint32_t warp = blockIdx.x * (kThreads / 32) + (tid >> 5);
  const PipeCtx b{soups, pb.error, pb.wait_limit_ns, pb.tune};
  const PipeQueue q = pb.queue;
  Server<L, kLanes> server(smem, tables, tid);
  Lane ln;
  ln.begin();
  if (lane >= server.kWidth) ln.state = kExhausted;
  // A warp serves the queue until every lane has claimed past its last task.
  while (true) {
    const bool progressed = server.iterate(b, q, ln, lane, warp % kCountSlots);
    if (__all_sync(0xffffffffu, ln.state == kExhausted)) return;
    if (!__any_sync(0xffffffffu, progressed)) __nanosleep(200);
  }
}

template <int L, int kWhich>
PipeKernel pipe_kernel() {
  constexpr uint32_t kLanes = pipe_widths(L).width[kWhich].pairs;
  static_assert(Server<L, kLanes>::kWidth == kLanes);
  return {reinterpret_cast<const void *>(&pipeline_kernel<L, kLanes>),
          server_bytes<L, kLanes>() + 512};
}

// The kernels of language L.
template <int L>
PipeKernels pipe_kernels() {
  PipeKernels k{};
  k.kernel[0] = pipe_kernel<L, 0>();
  if constexpr (pipe_widths(L).count > 1) k.kernel[1] = pipe_kernel<L, 1>();
  if constexpr (pipe_widths(L).count > 2) k.kernel[2] = pipe_kernel<L, 2>();
  return k;
}

}  // namespace
}  // namespace cubff

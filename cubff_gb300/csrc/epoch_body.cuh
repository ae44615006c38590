// epoch_body.cuh — the kernels of one epoch of one soup
// (MutateAndRunPrograms, common_language.h:157-193).
#pragma once

#include "internal.h"
#include "staged.cuh"

namespace cubff {

constexpr int kThreads = 128;  // one group of four warps
constexpr int kGroups = kThreads / 128;

// Shared memory per CTA.  SUBLEQ: two per-lane 128-byte areas per thread (the
// tape and the cycle check's snapshot); the staged languages: their warps', then
// the op and command tables.
template <uint32_t kWidth = 32>
struct SubleqMem {  // of a warp, kWidth lanes of which hold pairs
  uint32_t tapes[kPair / 4 * kWidth], snaps[kPair / 4 * kWidth];
};
// The pairs of a block that go on past their first stage.
template <int L, uint32_t kWidth>
struct LongPairs {
  static constexpr uint32_t kPairs = kThreads / 32 * kWidth;
  typename Stages<L>::State state[kPairs];  // by warp and lane
  uint32_t list[kPairs];
  uint32_t count, claimed;
};
template <int L, uint32_t kWidth = 8>
constexpr size_t epoch_smem_bytes() {
  if constexpr (LangTraits<L>::kStaged)
    return kThreads / 32 * sizeof(StagedMem<L, kWidth>) + 512 + sizeof(LongPairs<L, kWidth>);
  else return kThreads / 32 * sizeof(SubleqMem<>);
}

__device__ __forceinline__ void load_pair(const uint8_t *soup, uint32_t p1, uint32_t p2,
                                          uint32_t w[32]) {
  const uint4 *g1 = reinterpret_cast<const uint4 *>(soup + uint64_t(p1) * kTape);
  const uint4 *g2 = reinterpret_cast<const uint4 *>(soup + uint64_t(p2) * kTape);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint4 a = __ldcg(g1 + q);
    const uint4 b = __ldcg(g2 + q);
    w[4 * q + 0] = a.x; w[4 * q + 1] = a.y; w[4 * q + 2] = a.z; w[4 * q + 3] = a.w;
    w[16 + 4 * q + 0] = b.x; w[16 + 4 * q + 1] = b.y;
    w[16 + 4 * q + 2] = b.z; w[16 + 4 * q + 3] = b.w;
  }
}

// The pair back: first half, then second half (common_language.h:188-191; of a
// program paired with itself the second half stays).
__device__ __forceinline__ void store_pair(uint8_t *soup, uint32_t p1, uint32_t p2,
                                           const uint32_t w[32]) {
  uint4 *g1 = reinterpret_cast<uint4 *>(soup + uint64_t(p1) * kTape);
  uint4 *g2 = reinterpret_cast<uint4 *>(soup + uint64_t(p2) * kTape);
#pragma unroll
  for (int q = 0; q < 4; q++)
    g1[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
#pragma unroll
  for (int q = 0; q < 4; q++)
    g2[q] = make_uint4(w[16 + 4 * q], w[16 + 4 * q + 1], w[16 + 4 * q + 2], w[16 + 4 * q + 3]);
}

// Sets the bytes of the 32 draws from key0 on that mutate: set(b, byte).
template <class F>
__device__ __forceinline__ void mutate(uint64_t key0, uint32_t prob, F set) {
  uint32_t bits = mutation_word(key0, prob);
  while (bits) {
    const int b = __ffs(bits) - 1;
    bits &= bits - 1;
    set(b, static_cast<uint32_t>(splitmix64(key0 + b)) & 0xFFu);
  }
}

__device__ __forceinline__ void add_counts(const EpochArgs &a, uint32_t ops, uint32_t raw) {
  const uint32_t wops = __reduce_add_sync(0xffffffffu, ops);
  const uint32_t wraw = __reduce_add_sync(0xffffffffu, raw);
  if ((threadIdx.x & 31) == 0) {
    if (wops) atomicAdd(a.ops, static_cast<unsigned long long>(wops));
    if (a.raw && wraw) atomicAdd(a.raw, static_cast<unsigned long long>(wraw));
  }
}

// SUBLEQ: one pair per thread.
template <int L>
__global__ void __launch_bounds__(kThreads) epoch_kernel(EpochArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t tid = threadIdx.x;
  const uint64_t npairs = a.n / 2;
  const uint64_t k = uint64_t(blockIdx.x) * kThreads + tid;
  const bool active = k < npairs;
  SubleqMem<> &mem = reinterpret_cast<SubleqMem<> *>(smem)[tid >> 5];
  const LaneWords<32> t{reinterpret_cast<uint8_t *>(mem.tapes), tid & 31};
  const LaneWords<32> snap{reinterpret_cast<uint8_t *>(mem.snaps), tid & 31};

  uint32_t ops = 0;  // (SUBLEQ counts every step)
  if (active) {
    const uint32_t p1 = a.perm[2 * k], p2 = a.perm[2 * k + 1];
    uint32_t w[32];
    load_pair(a.soup, p1, p2, w);
#pragma unroll
    for (int q = 0; q < 32; q++) t.word(q) = w[q];
    const uint64_t key0 = (a.n * a.epoch_key + k) * kPair;
#pragma unroll 1
    for (int q = 0; q < kPair; q += 32)
      mutate(key0 + q, a.mutation_prob, [&](int i, uint32_t v) { t.set(q + i, v); });
    const uint64_t num_indices = a.d_num_indices ? *a.d_num_indices : a.num_indices;
    if (k < num_indices) {
      SubleqMachine<(L == kRsubleq4)> m;
      m.begin();
      while (!m.step(t, snap)) {
      }
      ops = m.ops();
    }
#pragma unroll
    for (int q = 0; q < 32; q++) w[q] = t.word(q);
    store_pair(a.soup, p1, p2, w);
  }
  add_counts(a, ops, ops);
}

// The staged languages.  A warp takes kWidth consecutive pairs: all lanes load
// and mutate them together, 8 pairs at a time (32 of their draws per lane), its
// first lanes run the first part of one each, and, where most of them go on and
// lanes may (Stages), all of it.  The other pairs that go on run on whole warps:
// those of a block wherever one is free, as the launch lasts as long as its slowest
// warp.  (One epoch of 2^17 programs evolved for 4096: forthtrivial 1.2 ms, bff8
// 1.6, bff 1.65; with 8 pairs to a warp, all run by that warp one after the other,
// 21, 7.0 and 1.9; one pair a lane 0.75, 1.1 and 1.25.)
template <int L, uint32_t kWidth>
__global__ void __launch_bounds__(kThreads, kWidth == 8 ? 5 : 4) staged_epoch_kernel(EpochArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  using LaneM = typename Stages<L>::Lane;
  uint8_t *tables = smem + kThreads / 32 * sizeof(StagedMem<L, kWidth>);
  const uint8_t *optab = tables, *cmdflag = tables + 256;
  LongPairs<L, kWidth> &longs = *reinterpret_cast<LongPairs<L, kWidth> *>(tables + 512);
  if (threadIdx.x == 0) longs.count = longs.claimed = 0;
  fill_tables<L>(tables);
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t npairs = a.n / 2;
  const uint64_t k0 = (uint64_t(blockIdx.x) * (kThreads / 32) + warp) * kWidth;
  const uint32_t count =
      k0 >= npairs ? 0 : static_cast<uint32_t>(npairs - k0 < kWidth ? npairs - k0 : kWidth);
  StagedMem<L, kWidth> *mems = reinterpret_cast<StagedMem<L, kWidth> *>(smem);
  StagedMem<L, kWidth> &mem = mems[warp];
  const LaneWords<kWidth> t = mem.tape(lane), stk = mem.stack(lane);
  uint32_t *soup = reinterpret_cast<uint32_t *>(a.soup);

  // Lane l holds word l of each pair: program `mine` of it, word l % 16.
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < count; j0 += 8) {
    uint32_t mine[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; j++)
      mine[j] = j0 + j < count ? a.perm[2 * (k0 + j0 + j) + (lane >> 4)] : 0;
#pragma unroll
    for (uint32_t j = 0; j < 8; j++)
      if (j0 + j < count)
        mem.tapes[lane * kWidth + j0 + j] = soup[uint64_t(mine[j]) * 16 + (lane & 15)];
    __syncwarp();
    // Mutations: lane l draws for 32 bytes of pair l / 4.
    const uint32_t j = j0 + lane / 4;
    if (j < count) {
      const uint32_t q = lane % 4 * 32;
      mutate((a.n * a.epoch_key + k0 + j) * kPair + q, a.mutation_prob,
             [&](int i, uint32_t v) { mem.tape(j).set(q + i, v); });
    }
  }
  __syncwarp();
  const uint64_t num_indices = a.d_num_indices ? *a.d_num_indices : a.num_indices;
  LaneM m;
  m.status = LaneM::kEnds;
  Mask128 cmd{0, 0};
  if (L <= kBffSelfmove) {
    for (uint32_t j = 0; j < count; j++) {
      const LaneWords<kWidth> tj = mem.tape(j);
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        w[q] = __ballot_sync(0xffffffffu, cmdflag[tj.get(32 * q + lane)] != 0);
      if (lane == j)
        cmd = Mask128{w[0] | static_cast<uint64_t>(w[1]) << 32, w[2] | static_cast<uint64_t>(w[3]) << 32};
    }
  }
  const bool evaluated = lane < count && k0 + lane < num_indices;
  if (evaluated) m.begin(t, cmd, optab);
  while (true) {
    const bool go = evaluated && m.status == LaneM::kRuns;
    if (!__any_sync(0xffffffffu, go)) break;
    if (go) m.step(t, stk, optab);
  }
  uint32_t ops = 0, raw = 0;
  if (evaluated && m.status == LaneM::kJumps) m.resolve(t, optab);
  // (bff8: 8 lanes are too few to be worth their dearer steps here.)
  if constexpr (Stages<L>::kCrowds && (kWidth > 8 || L > kBffSelfmove)) {
    constexpr int kCrowd = Stages<L>::crowd(kWidth);
    const bool goes_on = evaluated && m.status == LaneM::kJumps;
    if (__popc(__ballot_sync(0xffffffffu, goes_on)) >= kCrowd && goes_on) {
      LaneM::begin_cycle(mem.cycles[lane]);
      while (m.status != LaneM::kEnds) m.step_on(t, stk, optab, mem.cycles[lane]);
    }
  }
  if (evaluated && m.status == LaneM::kJumps) {
    longs.state[warp * kWidth + lane] = m.state();
    longs.list[atomicAdd(&longs.count, 1u)] = warp * kWidth + lane;
  } else if (evaluated) {
    ops = m.ops();
    raw = m.raw();
  }
  __syncthreads();
  while (true) {
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(&longs.claimed, 1u);
    next = __shfl_sync(0xffffffffu, next, 0);
    if (next >= longs.count) break;
    const uint32_t pair = longs.list[next], src = pair % kWidth;
    StagedMem<L, kWidth> &of = mems[pair / kWidth];
    const Counts c = run_on_warp<L>(mem.warp, of, src, longs.state[pair], lane, optab);
    of.tapes[lane * kWidth + src] = reinterpret_cast<const uint32_t *>(mem.warp.T)[lane];
    if (lane == 0) {
      ops += c.ops;
      raw += c.raw;
    }
  }
  __syncthreads();
  // First half, then second half (common_language.h:188-191): of a program
  // paired with itself the second half stays.
#pragma unroll 8
  for (uint32_t j = 0; j < count; j++) {
    const uint32_t mine = a.perm[2 * (k0 + j) + (lane >> 4)];
    const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 16);
    if (lane >= 16 || mine != other)
      soup[uint64_t(mine) * 16 + (lane & 15)] = mem.tapes[lane * kWidth + j];
  }
  add_counts(a, ops, raw);
}

}  // namespace cubff

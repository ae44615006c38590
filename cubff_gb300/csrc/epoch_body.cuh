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
struct SubleqMem {  // of a warp
  uint32_t tapes[kPair / 4 * 32], snaps[kPair / 4 * 32];
};
template <int L>
constexpr size_t epoch_smem_bytes() {
  if constexpr (LangTraits<L>::kStaged) return kThreads / 32 * sizeof(StagedMem<L>) + 512;
  else return kThreads / 32 * sizeof(SubleqMem);
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
  SubleqMem &mem = reinterpret_cast<SubleqMem *>(smem)[tid >> 5];
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
// and mutate them together (32 of their draws per lane),
// its first lanes run the first part of one each, and the pairs that go on run
// on the whole warp one after the other.  The launch lasts as long as its
// longest pairs, so a warp holds few.
template <int L>
__global__ void __launch_bounds__(kThreads, 5) staged_epoch_kernel(EpochArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  using LaneM = typename Stages<L>::Lane;
  constexpr uint32_t kWidth = StagedMem<L>::kWidth;
  uint8_t *tables = smem + kThreads / 32 * sizeof(StagedMem<L>);
  const uint8_t *optab = tables, *cmdflag = tables + 256;
  fill_tables<L>(tables);
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t npairs = a.n / 2;
  const uint64_t k0 = (uint64_t(blockIdx.x) * (kThreads / 32) + warp) * kWidth;
  if (k0 >= npairs) return;
  const uint32_t count = static_cast<uint32_t>(npairs - k0 < kWidth ? npairs - k0 : kWidth);
  StagedMem<L> &mem = reinterpret_cast<StagedMem<L> *>(smem)[warp];
  const LaneWords<kWidth> t = mem.tape(lane), stk = mem.stack(lane);
  uint32_t *soup = reinterpret_cast<uint32_t *>(a.soup);

  // Lane l holds word l of each pair: program `mine` of it, word l % 16.
  uint32_t mine[kWidth];
#pragma unroll
  for (uint32_t j = 0; j < kWidth; j++)
    mine[j] = j < count ? a.perm[2 * (k0 + j) + (lane >> 4)] : 0;
#pragma unroll
  for (uint32_t j = 0; j < kWidth; j++)
    if (j < count) mem.tapes[lane * kWidth + j] = soup[uint64_t(mine[j]) * 16 + (lane & 15)];
  __syncwarp();
  // Mutations: lane l draws for 32 bytes of pair l / 4.
  static_assert(kWidth * 4 == 32);
  if (lane / 4 < count) {
    const uint32_t q = lane % 4 * 32;
    mutate((a.n * a.epoch_key + k0 + lane / 4) * kPair + q, a.mutation_prob,
           [&](int i, uint32_t v) { mem.tape(lane / 4).set(q + i, v); });
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
  uint32_t longs = __ballot_sync(0xffffffffu, evaluated && m.status == LaneM::kJumps);
  if (evaluated && m.status == LaneM::kEnds) {
    ops = m.ops();
    raw = m.raw();
  }
  while (longs) {
    const uint32_t src = static_cast<uint32_t>(__ffs(longs) - 1);
    longs &= longs - 1;
    const Counts c = run_on_warp(mem, m, src, lane, optab);
    mem.tapes[lane * kWidth + src] = reinterpret_cast<const uint32_t *>(mem.warp.T)[lane];
    if (lane == src) {
      ops = c.ops;
      raw = c.raw;
    }
  }
  __syncwarp();
  // First half, then second half (common_language.h:188-191): of a program
  // paired with itself the second half stays.
#pragma unroll
  for (uint32_t j = 0; j < kWidth; j++) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, mine[j], 16);
    if (j < count && (lane >= 16 || mine[j] != other))
      soup[uint64_t(mine[j]) * 16 + (lane & 15)] = mem.tapes[lane * kWidth + j];
  }
  add_counts(a, ops, raw);
}

}  // namespace cubff

// epoch.cu — the fused epoch kernel (gather -> mutate -> run -> split -> count)
// and the soup-init, self-replication and histogram kernels, for all 13
// languages.
//
// The op count is reduced per warp (redux) and added with one atomic per warp,
// as IncreaseInsnCount does (common_language.h:56-63).
#include <algorithm>
#include <atomic>
#include <cstring>
#include "internal.h"
#include "epoch_body.cuh"

namespace cubff {
namespace {

// InitPrograms (common_language.h:138-155): one thread per 16-byte chunk.
__global__ void init_kernel(uint8_t *soup, uint64_t n, uint64_t key, int zero_init,
                            uint64_t count) {
  const uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= count * 4) return;
  const uint64_t idx = c >> 2;
  const uint64_t base = kTape * n * key + kTape * idx + (c & 3) * 16;
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t x = 0;
    if (!zero_init) {
#pragma unroll
      for (int b = 0; b < 4; b++)
        x |= (static_cast<uint32_t>(splitmix64(base + 4 * q + b)) & 0xFFu) << (8 * b);
    }
    v[q] = x;
  }
  reinterpret_cast<uint4 *>(soup)[c] = make_uint4(v[0], v[1], v[2], v[3]);
}

// CheckSelfRep (common_language.h:203-277): per program, 13 noise partners
// x (1 + 4) generations, then the byte-stability vote.
constexpr int kIters = 13, kGens = 4;

// Byte j of noise partner `it`.
__device__ __forceinline__ uint32_t noise(uint64_t local_seed, int it, uint32_t j) {
  return static_cast<uint32_t>(
             splitmix64(local_seed ^ splitmix64(uint64_t(it + 1) * kTape + j))) & 0xFF;
}

// Whether position i of the 13 final tapes counts for the program.
__device__ __forceinline__ bool stable(const uint8_t (*fin)[kPair], const uint8_t *prog, int i) {
  for (int x = 0; x < kIters; x++) {
    if (i < kTape && fin[x][i] != prog[i]) continue;
    uint32_t cnt = 1;
    for (int y = x + 1; y < kIters; y++) cnt += fin[x][i] == fin[y][i];
    if (cnt > kIters / 4) return true;
  }
  return false;
}

// SUBLEQ: one thread per program, its working tape in the shared-memory
// layout, its 13 final tapes in thread-local memory.
template <int L>
__global__ void __launch_bounds__(kThreads) selfrep_kernel(const uint8_t *soup,
                                                           uint64_t epoch_key,
                                                           uint64_t n, uint64_t count,
                                                           uint64_t *result) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t tid = threadIdx.x;
  const uint64_t index = uint64_t(blockIdx.x) * kThreads + tid;
  if (index >= count) return;
  const LaneBytes t{smem, lane_base(tid)};
  const LaneBytes stk{smem + kGroups * kGroupBytes, lane_base(tid)};
  uint8_t fin[kIters][kPair];
  const uint8_t *prog = soup + index * kTape;
  const uint64_t local_seed = splitmix64(n * epoch_key + index);
  for (int it = 0; it < kIters; it++) {
    for (int g = 0; g <= kGens; g++) {
      for (int j = 0; j < kTape; j++) {
        t.set(j, g == 0 ? prog[j] : t.get(kTape + j));
        t.set(kTape + j, noise(local_seed, it, j));
      }
      uint32_t raw;
      evaluate<L>(t, stk, nullptr, &raw);
    }
    for (int j = 0; j < kPair; j++) fin[it][j] = static_cast<uint8_t>(t.get(j));
  }
  uint64_t res[2] = {0, 0};
  for (int i = 0; i < kPair; i++) res[i / kTape] += stable(fin, prog, i);
  result[index] = res[0] < res[1] ? res[0] : res[1];
}

// The staged languages.  The 13 chains of 5 evaluations of a program are
// independent, and a chain of a self-replicator takes a whole warp some 0.2 ms;
// so a block takes kScored programs, its warps claim their chains one by one and
// keep the final tapes in shared memory, and all threads vote, one position
// each.  (One thread per program, 65 evaluations in a row, had a warp wait for
// the slowest of its 32 programs 65 times: 103 ms for a soup of 2^14 bff
// programs with self-replicators about; now 35.)
constexpr int kScored = 4;

// The chains of a program on the lanes of a warp.
template <int L>
struct ChainMem {
  static constexpr uint32_t kLanes = 16;
  uint32_t tapes[kLanes * kPair / 4];
  uint32_t stacks[Stages<L>::kStack ? kLanes * kPair / 4 : 4];
  typename Stages<L>::Lane::Cycle cycles[kLanes];
};

template <int L>
struct ScoreMem {
  typename Stages<L>::Mem warps[kThreads / 32];
  uint8_t fin[kScored][kIters][kPair];
  uint8_t prog[kScored][kTape];
  ChainMem<L> chains[Stages<L>::kCrowds ? kScored : 1];
  uint32_t votes[kScored][2];
  uint32_t claimed, left;
  uint8_t list[kScored * kIters];  // chains left for whole warps
  uint8_t tables[512];
};

// The 13 chains of program p, a lane each, if in the first generation so many of
// them go on past their first stage (Stages) that it is worth it; false if not.
// (2^13 forthtrivial programs evolved for 2112 epochs: 9.6 ms, chain by chain on
// whole warps 107, one program a lane 44; random ones, which gain nothing by it:
// 5.8, 4.0 and 24.)
template <int L>
__device__ __noinline__ bool chains_on_lanes(ScoreMem<L> &sm, uint32_t p, uint64_t local_seed,
                                             uint32_t lane) {
  using LaneM = typename Stages<L>::Lane;
  constexpr uint32_t kLanes = ChainMem<L>::kLanes;
  constexpr int kCrowd = Stages<L>::crowd(kIters);
  ChainMem<L> &mem = sm.chains[p];
  const bool mine = lane < kIters;
  const uint32_t it = mine ? lane : 0;
  const uint8_t *optab = sm.tables, *cmdflag = sm.tables + 256;
  const LaneWords<kLanes> t{reinterpret_cast<uint8_t *>(mem.tapes), it};
  const LaneWords<kLanes> stk{reinterpret_cast<uint8_t *>(mem.stacks), it};
  // (The partner's bytes wait where the final tape's second half will be.)
  uint32_t *fin = reinterpret_cast<uint32_t *>(sm.fin[p][it]);
  const uint32_t *prog = reinterpret_cast<const uint32_t *>(sm.prog[p]);
  if (mine)
    for (uint32_t j = 0; j < kTape; j++)
      sm.fin[p][it][kTape + j] = static_cast<uint8_t>(noise(local_seed, it, j));
  LaneM m;
  m.status = LaneM::kEnds;
  for (int g = 0; g <= kGens; g++) {
    if (mine) {
      for (uint32_t q = 0; q < kTape / 4; q++) {
        t.word(q) = g == 0 ? prog[q] : t.word(kTape / 4 + q);
        t.word(kTape / 4 + q) = fin[kTape / 4 + q];
      }
      Mask128 cmd{0, 0};
      if (L <= kBffSelfmove)
        for (int b = 0; b < kPair; b++) mask_assign(cmd, b, cmdflag[t.get(b)] != 0);
      m.begin(t, cmd, optab);
    }
    while (__any_sync(0xffffffffu, m.status == LaneM::kRuns))
      if (m.status == LaneM::kRuns) m.step(t, stk, optab);
    if (m.status == LaneM::kJumps) m.resolve(t, optab);
    const bool goes_on = m.status == LaneM::kJumps;
    const int going = __popc(__ballot_sync(0xffffffffu, goes_on));
    if (g == 0 && going < kCrowd) return false;
    if (goes_on) {
      LaneM::begin_cycle(mem.cycles[it]);
      while (m.status != LaneM::kEnds) m.step_on(t, stk, optab, mem.cycles[it]);
    }
    __syncwarp();
  }
  if (mine)
    for (uint32_t q = 0; q < kPair / 4; q++) fin[q] = t.word(q);
  return true;
}

template <int L>
__global__ void __launch_bounds__(kThreads, 5) staged_selfrep_kernel(const uint8_t *soup,
                                                                     uint64_t epoch_key,
                                                                     uint64_t n, uint64_t count,
                                                                     uint64_t *result) {
  extern __shared__ __align__(16) uint8_t smem[];
  ScoreMem<L> &sm = *reinterpret_cast<ScoreMem<L> *>(smem);
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint64_t first = uint64_t(blockIdx.x) * kScored;
  const uint32_t programs = static_cast<uint32_t>(count - first < kScored ? count - first : kScored);
  fill_tables<L>(sm.tables);
  for (uint32_t b = tid; b < programs * kTape; b += kThreads)
    sm.prog[0][b] = soup[first * kTape + b];
  if (tid < 2 * kScored) sm.votes[0][tid] = 0;
  if (tid == 0) sm.claimed = sm.left = 0;
  __syncthreads();
  if constexpr (Stages<L>::kCrowds) {
    static_assert(kScored == kThreads / 32);
    const uint32_t p = tid >> 5;
    if (p < programs && !chains_on_lanes(sm, p, splitmix64(n * epoch_key + first + p), lane) &&
        lane < kIters)
      sm.list[atomicAdd(&sm.left, 1u)] = static_cast<uint8_t>(p * kIters + lane);
    __syncthreads();
  }
  const uint32_t chains = Stages<L>::kCrowds ? sm.left : programs * kIters;
  typename Stages<L>::Mem &mem = sm.warps[tid >> 5];
  while (true) {
    uint32_t chain = 0;
    if (lane == 0) chain = atomicAdd(&sm.claimed, 1u);
    chain = __shfl_sync(0xffffffffu, chain, 0);
    if (chain >= chains) break;
    if (Stages<L>::kCrowds) chain = sm.list[chain];
    const uint32_t p = chain / kIters, it = chain % kIters;
    const uint64_t local_seed = splitmix64(n * epoch_key + first + p);
    const uint32_t n0 = noise(local_seed, it, lane), n1 = noise(local_seed, it, 32 + lane);
    for (int g = 0; g <= kGens; g++) {
      const uint8_t *from = g == 0 ? sm.prog[p] : mem.T + kTape;
      const uint8_t b0 = from[lane], b1 = from[32 + lane];
      __syncwarp();
      mem.T[lane] = b0;
      mem.T[32 + lane] = b1;
      mem.T[kTape + lane] = static_cast<uint8_t>(n0);
      mem.T[kTape + 32 + lane] = static_cast<uint8_t>(n1);
      __syncwarp();
      typename Stages<L>::template Warp<DeviceWarp> wm(DeviceWarp{lane}, mem, sm.tables);
      wm.run(wm.start(L == kBff || L == kBffPerm || L == kBff8 || L == kBffSelfmove));
      __syncwarp();
    }
    reinterpret_cast<uint32_t *>(sm.fin[p][it])[lane] =
        reinterpret_cast<const uint32_t *>(mem.T)[lane];
    __syncwarp();
  }
  __syncthreads();
  for (uint32_t p = 0; p < programs; p++)
    if (stable(sm.fin[p], sm.prog[p], static_cast<int>(tid)))
      atomicAdd(&sm.votes[p][tid / kTape], 1u);
  __syncthreads();
  if (tid < programs) {
    const uint32_t a = sm.votes[tid][0], b = sm.votes[tid][1];
    result[first + tid] = a < b ? a : b;
  }
}

// One evaluation of one tape: the call's latency is all there is (the kernel
// takes 8 us of it for a short program), so the tape comes with the launch and
// one copy brings back the result: 27 us a call of a bff tape.  (As an epoch of one
// pair in a buffer of the call's own, with two copies in, a memset and two copies
// out: 156.)
struct EvalTape {
  uint32_t words[kPair / 4];
};
struct EvalResult {
  uint32_t words[kPair / 4];
  uint32_t ops, raw;
};
// Results of calls under way, `kEvalSlots` at most; a call takes one for its own.
constexpr int kEvalSlots = 16;
__device__ EvalResult g_eval_results[kEvalSlots];

// One warp: as a pair of an epoch, with the other lanes' places empty.  The
// result goes to *out, or to the slot if out is null.
template <int L>
__global__ void __launch_bounds__(32)
    eval_kernel(const __grid_constant__ EvalTape tape, int slot, EvalResult *out) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t lane = threadIdx.x;
  EvalResult &res = out ? *out : g_eval_results[slot];
  if constexpr (LangTraits<L>::kStaged) {
    constexpr uint32_t kWidth = StagedMem<L>::kWidth;
    StagedMem<L> &mem = *reinterpret_cast<StagedMem<L> *>(smem);
    uint8_t *tables = smem + sizeof(StagedMem<L>);
    const uint8_t *optab = tables, *cmdflag = tables + 256;
    fill_tables<L>(tables);
    mem.tapes[lane * kWidth] = tape.words[lane];
    __syncwarp();
    const LaneWords<kWidth> t = mem.tape(0), stk = mem.stack(0);
    Mask128 cmd{0, 0};
    if (L <= kBffSelfmove) {
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        w[q] = __ballot_sync(0xffffffffu, cmdflag[t.get(32 * q + lane)] != 0);
      cmd = Mask128{w[0] | static_cast<uint64_t>(w[1]) << 32, w[2] | static_cast<uint64_t>(w[3]) << 32};
    }
    using LaneM = typename Stages<L>::Lane;
    LaneM m;
    m.status = LaneM::kEnds;
    if (lane == 0) {
      m.begin(t, cmd, optab);
      while (m.status == LaneM::kRuns) m.step(t, stk, optab);
      if (m.status == LaneM::kJumps) m.resolve(t, optab);
    }
    if (__any_sync(0xffffffffu, m.status == LaneM::kJumps)) {
      const Counts c = run_on_warp<L>(mem.warp, mem, 0, broadcast(m.state(), 0), lane, optab);
      res.words[lane] = reinterpret_cast<const uint32_t *>(mem.warp.T)[lane];
      if (lane == 0) {
        res.ops = c.ops;
        res.raw = c.raw;
      }
    } else {
      __syncwarp();
      res.words[lane] = mem.tapes[lane * kWidth];
      if (lane == 0) {
        res.ops = m.ops();
        res.raw = m.raw();
      }
    }
  } else {
    SubleqMem<> &mem = *reinterpret_cast<SubleqMem<> *>(smem);
    mem.tapes[lane * 32] = tape.words[lane];
    __syncwarp();
    if (lane == 0) {
      const LaneWords<32> t{reinterpret_cast<uint8_t *>(mem.tapes), 0};
      const LaneWords<32> snap{reinterpret_cast<uint8_t *>(mem.snaps), 0};
      SubleqMachine<(L == kRsubleq4)> m;
      m.begin();
      while (!m.step(t, snap)) {
      }
      res.ops = m.ops();
      res.raw = m.raw();
    }
    __syncwarp();
    res.words[lane] = mem.tapes[lane * 32];
  }
}

template <int L>
int launch_eval_t(const EvalTape &tape, int slot, EvalResult *out, cudaStream_t stream) {
  size_t smem = sizeof(SubleqMem<>);
  if constexpr (LangTraits<L>::kStaged) smem = sizeof(StagedMem<L>) + 512;
  eval_kernel<L><<<1, 32, smem, stream>>>(tape, slot, out);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

template <int L, uint32_t kWidth>
int launch_staged_epoch(const EpochArgs &a, uint64_t npairs, int device, cudaStream_t stream) {
  constexpr size_t smem = epoch_smem_bytes<L, kWidth>();
  if constexpr (smem > 48 << 10) {
    static std::atomic<uint64_t> raised;  // by device (zero-initialised)
    const uint64_t bit = 1ull << (device & 63);
    if (!(raised.load() & bit)) {
      CUBFF_CUDA_TRY(cudaFuncSetAttribute(staged_epoch_kernel<L, kWidth>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(smem)));
      raised.fetch_or(bit);
    }
  }
  constexpr uint64_t per_block = kThreads / 32 * kWidth;
  staged_epoch_kernel<L, kWidth>
      <<<static_cast<unsigned>((npairs + per_block - 1) / per_block), kThreads, smem, stream>>>(a);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

template <int L>
int launch_epoch_t(const EpochArgs &a, cudaStream_t stream) {
  const uint64_t npairs = a.n / 2;
  if (npairs == 0) return CUBFF_OK;
  if constexpr (LangTraits<L>::kStaged) {
    if constexpr (Stages<L>::kCrowds) {
      int device = 0, sms = 0;
      CUBFF_CUDA_TRY(cudaGetDevice(&device));
      CUBFF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
      // From 3 warps of 32 pairs per SM on, as in a pipelined launch.
      if (npairs >= uint64_t(sms) * 3 * 32) return launch_staged_epoch<L, 32>(a, npairs, device, stream);
      return launch_staged_epoch<L, 8>(a, npairs, device, stream);
    } else {
      return launch_staged_epoch<L, 8>(a, npairs, 0, stream);
    }
  } else {
    epoch_kernel<L><<<static_cast<unsigned>((npairs + kThreads - 1) / kThreads), kThreads,
                      epoch_smem_bytes<L>(), stream>>>(a);
    CUBFF_CUDA_TRY(cudaGetLastError());
    return CUBFF_OK;
  }
}

template <int L>
int launch_selfrep_t(const uint8_t *soup, uint64_t epoch_key, uint64_t n,
                     uint64_t count, uint64_t *result, cudaStream_t stream) {
  if (count == 0) return CUBFF_OK;
  if constexpr (LangTraits<L>::kStaged) {
    staged_selfrep_kernel<L><<<static_cast<unsigned>((count + kScored - 1) / kScored), kThreads,
                               sizeof(ScoreMem<L>), stream>>>(soup, epoch_key, n, count, result);
  } else {
    selfrep_kernel<L><<<static_cast<unsigned>((count + kThreads - 1) / kThreads), kThreads,
                        epoch_smem_bytes<L>(), stream>>>(soup, epoch_key, n, count, result);
  }
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

template <template <int> class F, typename... Args>
int dispatch_lang(int lang, Args &&...args) {
  switch (lang) {
    case kBff: return F<kBff>::run(args...);
    case kBffNoheads: return F<kBffNoheads>::run(args...);
    case kBffNoheads4bit: return F<kBffNoheads4bit>::run(args...);
    case kBffPerm: return F<kBffPerm>::run(args...);
    case kBff8: return F<kBff8>::run(args...);
    case kBff8Noheads: return F<kBff8Noheads>::run(args...);
    case kBffSelfmove: return F<kBffSelfmove>::run(args...);
    case kForth: return F<kForth>::run(args...);
    case kForthcopy: return F<kForthcopy>::run(args...);
    case kForthtrivial: return F<kForthtrivial>::run(args...);
    case kForthtrivialReset: return F<kForthtrivialReset>::run(args...);
    case kSubleq: return F<kSubleq>::run(args...);
    case kRsubleq4: return F<kRsubleq4>::run(args...);
  }
  return set_error(CUBFF_ENOTFOUND, "unknown language id %d", lang);
}

template <int L>
struct EpochLauncher {
  static int run(const EpochArgs &a, cudaStream_t s) { return launch_epoch_t<L>(a, s); }
};
template <int L>
struct EvalLauncher {
  static int run(const EvalTape &tape, int slot, EvalResult *out, cudaStream_t s) {
    return launch_eval_t<L>(tape, slot, out, s);
  }
};
template <int L>
struct SelfrepLauncher {
  static int run(const uint8_t *soup, uint64_t key, uint64_t n, uint64_t count,
                 uint64_t *result, cudaStream_t s) {
    return launch_selfrep_t<L>(soup, key, n, count, result, s);
  }
};

}  // namespace

int launch_epoch(int lang, const EpochArgs &a, cudaStream_t stream) {
  return dispatch_lang<EpochLauncher>(lang, a, stream);
}

int eval_pair(int lang, uint8_t *tape, uint64_t *ops, uint64_t *raw) {
  // The slots taken, by device (devices 64 apart share theirs).
  static std::atomic<uint32_t> taken[64];  // (zero-initialised: static storage)
  int device = 0;
  CUBFF_CUDA_TRY(cudaGetDevice(&device));
  std::atomic<uint32_t> &mine = taken[device & 63];
  uint32_t seen = mine.load();
  int slot = 0;
  do {
    for (slot = 0; slot < kEvalSlots && ((seen >> slot) & 1); slot++) {
    }
  } while (slot < kEvalSlots && !mine.compare_exchange_weak(seen, seen | (1u << slot)));
  EvalResult *out = nullptr;  // of this call, when all slots are taken
  if (slot == kEvalSlots) CUBFF_CUDA_TRY(cudaMalloc(&out, sizeof(EvalResult)));
  EvalTape in;
  EvalResult res;
  std::memcpy(in.words, tape, kPair);
  const cudaStream_t stream = nullptr;
  const int st = dispatch_lang<EvalLauncher>(lang, in, slot, out, stream);
  cudaError_t err = cudaSuccess;
  if (st == CUBFF_OK)
    err = out ? cudaMemcpy(&res, out, sizeof(res), cudaMemcpyDeviceToHost)
              : cudaMemcpyFromSymbol(&res, g_eval_results, sizeof(res), slot * sizeof(res));
  if (out) cudaFree(out);
  else mine.fetch_and(~(1u << slot));
  if (st != CUBFF_OK) return st;
  if (err != cudaSuccess) return set_error(CUBFF_EDEVICE, "eval_pair: %s", cudaGetErrorString(err));
  std::memcpy(tape, res.words, kPair);
  *ops = res.ops;
  if (raw) *raw = res.raw;
  return CUBFF_OK;
}

int launch_selfrep(int lang, const uint8_t *soup, uint64_t epoch_key, uint64_t n,
                   uint64_t count, uint64_t *result, cudaStream_t stream) {
  return dispatch_lang<SelfrepLauncher>(lang, soup, epoch_key, n, count, result, stream);
}

int launch_init(uint64_t key, uint64_t n, uint8_t *soup, int zero_init,
                uint64_t count, cudaStream_t stream) {
  if (count == 0) return CUBFF_OK;
  const uint64_t chunks = count * 4;
  const unsigned grid = static_cast<unsigned>((chunks + 255) / 256);
  init_kernel<<<grid, 256, 0, stream>>>(soup, n, key, zero_init, count);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

// Byte histogram of a soup (the statistics of common_language.h:519-533):
// per-block counters in shared memory, added into 256 global counters.
__global__ void histogram_kernel(const uint32_t *words, uint64_t n_words,
                                 unsigned long long *counts) {
  __shared__ uint32_t h[256];
  for (uint32_t c = threadIdx.x; c < 256; c += blockDim.x) h[c] = 0;
  __syncthreads();
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n_words;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t w = words[i];
    atomicAdd(&h[w & 0xFF], 1u);
    atomicAdd(&h[(w >> 8) & 0xFF], 1u);
    atomicAdd(&h[(w >> 16) & 0xFF], 1u);
    atomicAdd(&h[w >> 24], 1u);
  }
  __syncthreads();
  for (uint32_t c = threadIdx.x; c < 256; c += blockDim.x)
    if (h[c]) atomicAdd(&counts[c], static_cast<unsigned long long>(h[c]));
}

int launch_histogram(const uint8_t *soup, uint64_t n_bytes, unsigned long long *counts,
                     cudaStream_t stream) {
  CUBFF_CUDA_TRY(cudaMemsetAsync(counts, 0, 256 * sizeof(unsigned long long), stream));
  const uint64_t words = n_bytes / 4;  // soups are num_programs * 64 bytes
  if (words == 0) return CUBFF_OK;
  const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((words + 255) / 256, 1216));
  histogram_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uint32_t *>(soup), words,
                                               counts);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

}  // namespace cubff

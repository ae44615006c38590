// staged.cuh — running the two machines of a staged language (Stages, interp.cuh)
// in a warp's shared memory: what the pipelined, the per-epoch and the
// self-replication kernels share.
#pragma once

#include "interp.cuh"

namespace cubff {

// A warp's shared memory: the tapes (and stacks) of kWidth lanes, interleaved,
// and the warp machine's.
template <int L, uint32_t kLanes = 8>
struct StagedMem {
  static constexpr uint32_t kWidth = kLanes;  // lanes that hold pairs
  uint32_t tapes[kWidth * kPair / 4];
  uint32_t stacks[Stages<L>::kStack ? kWidth * kPair / 4 : 4];
  typename Stages<L>::Lane::Cycle cycles[Stages<L>::kCrowds ? kWidth : 1];
  typename Stages<L>::Mem warp;

  __device__ __forceinline__ LaneWords<kWidth> tape(uint32_t lane) {
    return {reinterpret_cast<uint8_t *>(tapes), lane};
  }
  __device__ __forceinline__ LaneWords<kWidth> stack(uint32_t lane) {
    return {reinterpret_cast<uint8_t *>(stacks), lane};
  }
};

__device__ __forceinline__ BffState broadcast(const BffState &s, uint32_t src) {
  constexpr uint32_t kAll = 0xffffffffu;
  BffState r;
  r.q = __shfl_sync(kAll, s.q, src);
  r.h0 = __shfl_sync(kAll, s.h0, src);
  r.h1 = __shfl_sync(kAll, s.h1, src);
  r.i = __shfl_sync(kAll, s.i, src);
  r.n = __shfl_sync(kAll, s.n, src);
  r.mods = __shfl_sync(kAll, s.mods, src);
  return r;
}
__device__ __forceinline__ ForthState broadcast(const ForthState &s, uint32_t src) {
  constexpr uint32_t kAll = 0xffffffffu;
  ForthState r;
  r.begin();
  r.pos = __shfl_sync(kAll, s.pos, src);
  r.sp = __shfl_sync(kAll, s.sp, src);
  r.r0 = __shfl_sync(kAll, s.r0, src);
  r.r1 = __shfl_sync(kAll, s.r1, src);
  r.i = __shfl_sync(kAll, s.i, src);
  r.nops = __shfl_sync(kAll, s.nops, src);
  r.mods = __shfl_sync(kAll, s.mods, src);
  return r;
}

struct Counts {
  uint32_t ops, raw, mods;
};

// Runs the pair of lane `src` of a warp's memory `of`, from state st, to its end on
// the whole warp; its tape is then in work.T.
template <int L, uint32_t kWidth>
__device__ __forceinline__ Counts run_on_warp(typename Stages<L>::Mem &work,
                                              const StagedMem<L, kWidth> &of, uint32_t src,
                                              const typename Stages<L>::State &st, uint32_t lane,
                                              const uint8_t *optab) {
  __syncwarp();  // the lane's tape
  reinterpret_cast<uint32_t *>(work.T)[lane] = of.tapes[lane * kWidth + src];
  if constexpr (Stages<L>::kStack)
    reinterpret_cast<uint32_t *>(work.stk)[lane] = of.stacks[lane * kWidth + src];
  __syncwarp();
  typename Stages<L>::template Warp<DeviceWarp> wm(DeviceWarp{lane}, work, optab);
  wm.run(st);
  __syncwarp();
  return {wm.ops(), wm.raw(), wm.mods()};
}

// Op table, and command flags (BFF: op < kNull) behind it.
template <int L>
__device__ __forceinline__ void fill_tables(uint8_t *tables) {
  for (uint32_t c = threadIdx.x; c < 256; c += blockDim.x) {
    tables[c] = op_of(L, c);
    tables[256 + c] = op_of(L, c) < kNull;
  }
}

}  // namespace cubff

// coop.cuh — what the warp-cooperative interpreters are written in: code that
// all 32 lanes run with the same values ("uniform"), and lane-wise parts given
// as functions of the lane number.  On the device a lane evaluates its own; on
// the host (tests) one thread evaluates all 32 in turn.
#pragma once

#include "cycle.cuh"

namespace cubff {

constexpr int kWarp = 32;

struct DeviceWarp {
  uint32_t lane;
  // One value per lane.
  template <class T>
  struct Lanes {
    T v;
    __device__ __forceinline__ T operator()(uint32_t) const { return v; }
  };
  template <class F>
  __device__ __forceinline__ auto map(F f) const -> Lanes<decltype(f(0u))> {
    return {f(lane)};
  }
  template <class F>
  __device__ __forceinline__ uint32_t ballot(F f) const {
    return __ballot_sync(0xffffffffu, f(lane));
  }
  template <class F>
  __device__ __forceinline__ bool any(F f) const {
    return __any_sync(0xffffffffu, f(lane));
  }
  template <class F>
  __device__ __forceinline__ void each(F f) const {
    f(lane);
  }
  // Orders the lanes' shared-memory accesses before against those after.
  __device__ __forceinline__ void sync() const { __syncwarp(); }
};

struct HostWarp {
  template <class T>
  struct Lanes {
    T v[kWarp];
    T operator()(uint32_t l) const { return v[l]; }
  };
  template <class F>
  auto map(F f) const -> Lanes<decltype(f(0u))> {
    Lanes<decltype(f(0u))> r;
    for (uint32_t l = 0; l < kWarp; l++) r.v[l] = f(l);
    return r;
  }
  template <class F>
  uint32_t ballot(F f) const {
    uint32_t m = 0;
    for (uint32_t l = 0; l < kWarp; l++) m |= static_cast<uint32_t>(f(l) ? 1u : 0u) << l;
    return m;
  }
  template <class F>
  bool any(F f) const {
    return ballot(f) != 0;
  }
  template <class F>
  void each(F f) const {
    for (uint32_t l = 0; l < kWarp; l++) f(l);
  }
  void sync() const {}
};

__host__ __device__ __forceinline__ int popc32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return __builtin_popcount(x);
#endif
}

// Lowest / highest set bit of a non-zero x.
__host__ __device__ __forceinline__ int low32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __ffs(static_cast<int>(x)) - 1;
#else
  return __builtin_ctz(x);
#endif
}
__host__ __device__ __forceinline__ int high32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return 31 - __clz(static_cast<int>(x));
#else
  return 31 - __builtin_clz(x);
#endif
}

}  // namespace cubff

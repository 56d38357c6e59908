// warp_stream.cuh -- what the row-streaming step kernels share: neighbour exchange along
// a warp's row of cells and asynchronous copies into a warp's staging area. Included
// inside a build's arithmetic namespace.
#pragma once

constexpr unsigned kFullWarp = 0xffffffffu;

// Whether any lane of the warp has `p` (VOTE: all of its lanes call), or this one.
template <bool VOTE>
__device__ __forceinline__ bool any_lane(bool p) {
  if constexpr (VOTE) return __any_sync(kFullWarp, p);
  return p;
}

// The value one cell to the west / east of this lane's (the outermost lanes get their own
// back: they hold halo cells whose results nobody stores).
__device__ __forceinline__ float west_of(float x) { return __shfl_up_sync(kFullWarp, x, 1); }
__device__ __forceinline__ float east_of(float x) { return __shfl_down_sync(kFullWarp, x, 1); }

// Asynchronous copy of this lane's word of array K of a staged row, or of a zero where
// CHECK and !ok (`safe` is any mapped address). Each lane copies, and after its own wait
// reads back, its own words only.
template <int K, bool CHECK>
__device__ __forceinline__ void copy_word(unsigned dst, const float* src, bool ok, const float* safe) {
  if constexpr (CHECK) {
    asm volatile("cp.async.ca.shared.global [%0+%2], [%1], 4, %3;" ::"r"(dst), "l"(ok ? src : safe), "n"(K * 128),
                 "r"(ok ? 4 : 0)
                 : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0+%2], [%1], 4;" ::"r"(dst), "l"(src), "n"(K * 128) : "memory");
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

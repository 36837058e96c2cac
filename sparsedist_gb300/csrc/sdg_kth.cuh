// sdg_kth.cuh -- the k-th largest of a float array in shared memory, found by
// a group of threads (a warp, or a block of several warps).
//
// The floats are compared through the order-preserving map onto uint32 and
// the answer's bits are fixed from the highest down: bit b stays set when at
// least k keys reach the prefix with it.  The search starts at the highest
// bit in which the largest and the smallest key differ, so values of similar
// magnitude need about 20 rounds of count / group-sum instead of k dependent
// sorted insertions.
#pragma once

#include <cstdint>

namespace sdg {
namespace kth {

// ascending float -> ascending key (-inf .. +inf; the caller has no NaN)
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fkey_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Group operations of WARPS warps: a single warp, or the whole block of
// WARPS * 32 threads (red: WARPS words of shared memory).
template <int WARPS>
struct Group {
  uint32_t* red;
  __device__ __forceinline__ int size() const { return WARPS * 32; }
  __device__ __forceinline__ int rank() const { return WARPS == 1 ? (threadIdx.x & 31) : threadIdx.x; }
  __device__ __forceinline__ void sync() const {
    if (WARPS == 1) __syncwarp(); else __syncthreads();
  }
  // every thread gets the sum; the group may write shared memory afterwards
  __device__ __forceinline__ uint32_t sum(uint32_t v) const {
    v = __reduce_add_sync(0xffffffffu, v);
    if (WARPS > 1) {
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
      __syncthreads();
      v = 0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) v += red[w];
      __syncthreads();
    }
    return v;
  }
  __device__ __forceinline__ uint32_t bit_or(uint32_t v) const {
    v = __reduce_or_sync(0xffffffffu, v);
    if (WARPS > 1) {
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
      __syncthreads();
      v = 0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) v |= red[w];
      __syncthreads();
    }
    return v;
  }
};

// The k-th largest of keys[0 .. n), 1 <= k <= n, written before a group sync.
template <int WARPS>
__device__ __forceinline__ uint32_t largest(const Group<WARPS>& g, const uint32_t* keys, int n, int k) {
  const uint32_t first = keys[0];
  uint32_t diff = 0;
  for (int i = g.rank(); i < n; i += g.size()) diff |= keys[i] ^ first;
  diff = g.bit_or(diff);
  if (!diff) return first;
  const int top = 31 - __clz((int)diff);
  // the bits above `top` are common to every key
  uint32_t ans = (top == 31) ? 0u : (first & ~((2u << top) - 1u));
  for (int b = top; b >= 0; --b) {
    const uint32_t t = ans | (1u << b);
    uint32_t c = 0;
    for (int i = g.rank(); i < n; i += g.size()) c += keys[i] >= t;
    if (g.sum(c) >= (uint32_t)k) ans = t;
  }
  return ans;
}

}  // namespace kth
}  // namespace sdg

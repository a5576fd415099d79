// warp_list.cuh -- a sorted list of uint64 keys distributed over the 32
// lanes of a warp (entry e lives in register slot e/32 of lane e%32), with
// ballot-based insertion, and bitonic sorts and merges of 32 keys.  Used by
// the fused top-k epilogues of the FP32 kernels and of the IVF list scan.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace mann {
namespace wl {

constexpr unsigned FULL = 0xFFFFFFFFu;

template <int KW>
__device__ __forceinline__ void list_insert(uint64_t (&L)[KW], uint64_t c, int lane) {
  int pos = 0;
#pragma unroll
  for (int s = 0; s < KW; ++s) pos += __popc(__ballot_sync(FULL, L[s] < c));
  uint64_t up[KW], last[KW];
#pragma unroll
  for (int s = 0; s < KW; ++s) {
    up[s] = __shfl_up_sync(FULL, L[s], 1);
    last[s] = __shfl_sync(FULL, L[s], 31);
  }
#pragma unroll
  for (int s = 0; s < KW; ++s) {
    const int e = s * 32 + lane;
    uint64_t shifted = up[s];
    if (lane == 0) shifted = (s == 0) ? KEY_NONE : last[s > 0 ? s - 1 : 0];
    if (e > pos) L[s] = shifted;
    else if (e == pos) L[s] = c;
  }
}

template <int KW>
__device__ __forceinline__ uint64_t list_get(const uint64_t (&L)[KW], int e) {
  const int slot = e >> 5, ln = e & 31;
  uint64_t v = L[0];
#pragma unroll
  for (int s = 1; s < KW; ++s)
    if (slot == s) v = L[s];
  return __shfl_sync(FULL, v, ln);
}

// One compare-exchange stage of a warp bitonic network (lane holds one key).
__device__ __forceinline__ uint64_t cmpex(uint64_t v, int j, bool keep_min) {
  const uint64_t o = __shfl_xor_sync(FULL, (unsigned long long)v, j);
  return keep_min == (o < v) ? o : v;
}

// Ascending sort of one key per lane.
__device__ __forceinline__ uint64_t sort32(uint64_t c, int lane) {
#pragma unroll
  for (int w = 2; w <= 32; w <<= 1)
#pragma unroll
    for (int j = w >> 1; j > 0; j >>= 1) c = cmpex(c, j, ((lane & j) == 0) == ((lane & w) == 0));
  return c;
}

// Whether key (each lane its own, not KEY_NONE) is an entry of the sorted
// ascending list of 32 keys that the lanes hold in `list`.
__device__ __forceinline__ bool contains32(uint64_t list, uint64_t key, int lane) {
  int at = 0;  // the last entry at or below key, or entry 0
#pragma unroll
  for (int w = 16; w > 0; w >>= 1)
    if (__shfl_sync(FULL, (unsigned long long)list, at + w) <= key) at += w;
  const uint64_t e = __shfl_sync(FULL, (unsigned long long)list, at);
  return e == key && key != KEY_NONE;
}

// Sorted ascending lists of 32 keys, one entry per lane: the 32 smallest of both.
__device__ __forceinline__ uint64_t merge32(uint64_t a, uint64_t b, int lane) {
  const uint64_t r = __shfl_sync(FULL, (unsigned long long)b, 31 - lane);
  uint64_t m = r < a ? r : a;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) m = cmpex(m, j, (lane & j) == 0);
  return m;
}

}  // namespace wl
}  // namespace mann

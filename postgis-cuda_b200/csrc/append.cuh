// Compaction in one kernel: the items that a block keeps go to consecutive places behind a counter, one atomic per
// APPEND_ITEMS items. Order is kept inside a block's items only, so it serves rows in no set order and keys that are sorted
// afterwards. Against flags, a device scan, a scatter and a read of the last sum: two launches and two small copies less
// per batch, and no flag and offset arrays. Compaction of 100 queries' rows 0.045 -> 0.024 ms, 2M points' keys with their
// sort 0.286 -> 0.172 ms, the 8 rounds of a 300k-parcel cluster 0.577 -> 0.46 ms.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gsj {

constexpr int APPEND_THREADS = 256, APPEND_ITEMS = 4 * APPEND_THREADS;
inline unsigned append_grid(uint64_t n) { return (unsigned)((n + APPEND_ITEMS - 1) / APPEND_ITEMS); }

// keep(i) for the block's items i < n, then put(i, place) for those kept; called by the whole block of APPEND_THREADS
template <class Keep, class Put>
__device__ __forceinline__ void append_items(uint64_t n, unsigned long long* counter, Keep&& keep, Put&& put) {
  __shared__ uint32_t s_off[APPEND_THREADS / 32];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t i0 = (uint64_t)blockIdx.x * APPEND_ITEMS + w * 128 + lane;   // a warp takes 128 consecutive items
  unsigned m[4];
  uint32_t mine = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint64_t i = i0 + q * 32;
    m[q] = __ballot_sync(0xffffffffu, i < n && keep(i));
    mine += __popc(m[q]);
  }
  if (lane == 0) s_off[w] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t sum = 0;
    for (int k = 0; k < APPEND_THREADS / 32; k++) { const uint32_t c = s_off[k]; s_off[k] = sum; sum += c; }
    s_base = sum ? atomicAdd(counter, (unsigned long long)sum) : 0ull;
  }
  __syncthreads();
  unsigned long long at = s_base + s_off[w];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if ((m[q] >> lane) & 1u) put(i0 + q * 32, at + __popc(m[q] & ((1u << lane) - 1)));
    at += __popc(m[q]);
  }
}

// pair keys in the fewest bits, for the radix sort: a above b, b in `bits` bits
inline int key_bits(uint64_t n) { int b = 1; while (b < 63 && (n - 1) >> b) b++; return b; }   // n >= 1 values
__device__ __forceinline__ unsigned long long pair_key(uint32_t a, uint32_t b, int bits) { return ((unsigned long long)a << bits) | b; }
__device__ __forceinline__ uint2 key_pair(unsigned long long k, int bits) { return make_uint2((uint32_t)(k >> bits), (uint32_t)(k & ((1ull << bits) - 1))); }

}  // namespace gsj

// The sample of the top-k threshold estimate and the selection of a rank among few keys, shared by the
// threshold kernel and the compress kernel that estimates for itself.
#pragma once
#include "cx_device.cuh"

namespace cx {

// element that sample i looks at (the reference's float arithmetic)
__device__ __forceinline__ int64_t sample_position(int i, int64_t n, int use_all, float stepsize) {
  if (use_all) return i;
  const int64_t pos = (int64_t)(int)__fmul_rn((float)i, stepsize);
  return pos > n - 1 ? n - 1 : pos;
}

// One warp, one key per lane, the first `count` lanes: the key of rank `rank` in descending order.
__device__ __forceinline__ uint32_t warp_rank(uint32_t key, int count, int lane, uint32_t rank) {
  uint32_t gt = 0, ge = 0;
  for (int j = 0; j < count; ++j) {
    const uint32_t other = __shfl_sync(0xffffffffu, key, j);
    gt += other > key ? 1u : 0u;
    ge += other >= key ? 1u : 0u;
  }
  const uint32_t who = __ballot_sync(0xffffffffu, lane < count && gt <= rank && rank < ge);
  return __shfl_sync(0xffffffffu, key, __ffs(who) - 1);
}

// One warp: the key of rank `rank` among s_keys[0, s), s <= 1024, entries up to 1024 zero; list: scratch
// of 1024 words.  As in the block-wide selection, the (rank + 1)-th largest of the lanes' maxima leaves
// few keys to rank for ranks below 32; otherwise bisection over the bits of 32 keys per lane.
__device__ __forceinline__ uint32_t warp_select(const uint32_t* s_keys, int s, uint32_t rank, int lane, uint32_t* list) {
  uint32_t k[32], mx = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) { k[j] = s_keys[32 * j + lane]; mx = max(mx, k[j]); }
  if (rank < 32) {
    const uint32_t bound = warp_rank(mx, 32, lane, rank);
    uint32_t left = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const bool in = 32 * j + lane < s && k[j] >= bound;
      const uint32_t who = __ballot_sync(0xffffffffu, in);
      if (in) list[left + __popc(who & ((1u << lane) - 1u))] = k[j];
      left += __popc(who);
    }
    __syncwarp();
    if (left <= 32) return warp_rank(lane < (int)left ? list[lane] : 0u, (int)left, lane, rank);
  }
  uint32_t t = 0;
  for (int bit = 30; bit >= 0; --bit) {
    const uint32_t c = t | (1u << bit);
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) n += k[j] >= c ? 1u : 0u;
    if (__reduce_add_sync(0xffffffffu, n) > rank) t = c;
  }
  return t;
}

}  // namespace cx

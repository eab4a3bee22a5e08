// uc_lookback.cuh — chained prefix sums inside one kernel: blocks take work
// items in order from a ticket counter, publish each item's sum, and a warp
// adds up the sums of the items before it (decoupled look-back, Merrill and
// Garland 2016).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace uc {

// One 64-bit word per item: the top two bits say what the other 62 hold
// (0: nothing yet, 1: the item's own sum, 2: the sum of all items up to it),
// so a reader needs no ordering against other memory.
constexpr unsigned long long LB_SUM = 1ull << 62, LB_PREFIX = 2ull << 62, LB_VALUE = (1ull << 62) - 1ull;
// Polls of one word before the wait gives up.  An item is published only by
// a block that runs (tickets are handed out in order), so the limit is
// reached only when something is broken.
constexpr uint32_t LB_POLLS = 1u << 22;

__device__ __forceinline__ void lb_publish(unsigned long long* st, uint32_t i, unsigned long long tag,
                                           unsigned long long v) {
  atomicExch(st + i, tag | v);
}

// Sum of the items before item i (every lane of one warp calls; item i's own
// sum is published already).  Publishes item i's inclusive prefix.  A wait that
// runs out sets `bit` in *fail; one that meets a failure (any bit) gives up.
__device__ __forceinline__ unsigned long long lb_exclusive(unsigned long long* st, uint32_t i,
                                                           unsigned long long own, uint32_t* fail,
                                                           uint32_t bit = 1u) {
  const uint32_t lane = threadIdx.x & 31u;
  unsigned long long sum = 0;
  int64_t j = int64_t(i) - 1;  // nearest item of the window of 32
  while (j >= 0) {
    const int64_t at = j - int64_t(lane);
    unsigned long long v = LB_PREFIX;  // before the first item: a prefix of 0
    if (at >= 0) {
      v = 0;
      for (uint32_t p = 0; p < LB_POLLS; ++p) {
        v = *reinterpret_cast<volatile unsigned long long*>(st + at);
        if (v) break;
        if ((p & 1023u) == 1023u && *reinterpret_cast<volatile uint32_t*>(fail)) break;
      }
      if (!v) {
        atomicOr(fail, bit);
        v = LB_PREFIX;
      }
    }
    const uint32_t pm = __ballot_sync(0xFFFFFFFFu, (v & LB_PREFIX) != 0);
    const uint32_t last = pm ? uint32_t(__ffs(pm)) - 1u : 31u;  // the nearest prefix ends the walk
    unsigned long long add = lane <= last ? (v & LB_VALUE) : 0ull;
#pragma unroll
    for (int o = 16; o; o >>= 1) add += __shfl_xor_sync(0xFFFFFFFFu, add, o);
    sum += add;
    if (pm) break;
    j -= 32;
  }
  if (lane == 0) lb_publish(st, i, LB_PREFIX, sum + own);
  return sum;
}

}  // namespace uc

// The shared-memory slots a warp copies row vectors into (wv_link.cu).  A copy
// is asynchronous, and two copies in flight have no order: a slot may be taken
// only when no copy into it is under way.  A slot given back before its copy
// was waited for is therefore kept apart until the next wait for all copies.
// Host code too, so that the rule can be checked without a device.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define WV_SLOTS_FN __host__ __device__ __forceinline__
#else
#define WV_SLOTS_FN inline
#endif

namespace wv {

struct Slots {
  unsigned long long free;     // not in use, no copy into them under way
  unsigned long long pending;  // given back; the copy into them may be under way

  WV_SLOTS_FN void reset(uint32_t count) {  // (1 to 64 slots)
    free = ~0ull >> (64 - count);
    pending = 0;
  }
  // wait(): returns once every copy started so far has landed
  template <class Wait>
  WV_SLOTS_FN void reclaim(Wait wait) {
    if (!pending) return;
    wait();
    free |= pending;
    pending = 0;
  }
  template <class Wait>
  WV_SLOTS_FN uint32_t take(Wait wait) {
    reclaim(wait);
#ifdef __CUDA_ARCH__
    const uint32_t f = (uint32_t)(__ffsll((long long)free) - 1);
#else
    const uint32_t f = (uint32_t)(__builtin_ffsll((long long)free) - 1);
#endif
    free &= free - 1;
    return f;
  }
  // a slot whose copy may not have landed
  WV_SLOTS_FN void give_back(uint32_t f) { pending |= 1ull << f; }
};

}  // namespace wv

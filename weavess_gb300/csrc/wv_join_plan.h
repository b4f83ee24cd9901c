// Which nodes of NN-Descent's local join run in one launch.  Host code only.
#pragma once
#include <algorithm>
#include <cstdint>

namespace wv {

// what one launch may hold: offers, and entries of its nodes' lists (each may
// need a descriptor, whose place is a 32-bit prefix sum over the targets)
struct JoinLimits {
  uint64_t offers, lists;
};
constexpr uint64_t JOIN_LISTS_MAX = 0xffffffffull;

// list entries whose descriptors (desc_bytes each) may be held: half of what is
// free or held by them already (the rest of a join needs memory too), and not
// below a million
inline uint64_t join_lists_room(uint64_t free_bytes, uint64_t held_bytes, uint64_t desc_bytes) {
  const uint64_t half = (free_bytes + held_bytes) / 2 / desc_bytes;
  return std::min(JOIN_LISTS_MAX, std::max({half, held_bytes / desc_bytes, (uint64_t)1 << 20}));
}

struct JoinChunk {
  uint32_t end;            // nodes [n0, end)
  uint64_t offers, lists;  // at most so many offers; list entries
};

// the most nodes from n0 on that stay within the limits, and at least one
// (which may exceed them: the caller looks)
inline JoinChunk join_chunk(const uint32_t *lnew, const uint32_t *lold, uint32_t n0, uint32_t n,
                            const JoinLimits &lim) {
  JoinChunk c{n0, 0, 0};
  while (c.end < n) {
    const uint64_t a = lnew[c.end], b = lold[c.end];
    const uint64_t ub = a * (a - (a > 0)) + 2 * a * b;  // 2 offers per pair
    const uint64_t ls = a ? a + b : 0;                  // (a node without new ids joins nothing)
    if (c.end > n0 && (c.offers + ub > lim.offers || c.lists + ls > lim.lists)) break;
    c.offers += ub;
    c.lists += ls;
    c.end++;
  }
  return c;
}

}  // namespace wv

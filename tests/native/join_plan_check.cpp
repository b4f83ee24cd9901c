// Checks weavess_gb300/csrc/wv_join_plan.h on made-up list lengths: the chunks
// cover all nodes in order, stay within both limits, and take as many nodes as
// they can.  Prints "OK <chunks>" or the first fault.
#include <cstdio>
#include <random>
#include <vector>

#include "../../weavess_gb300/csrc/wv_join_plan.h"

using namespace wv;

static long check(const std::vector<uint32_t> &a, const std::vector<uint32_t> &b, JoinLimits lim) {
  const uint32_t n = (uint32_t)a.size();
  auto offers = [&](uint32_t i) { return (uint64_t)a[i] * (a[i] ? a[i] - 1 : 0) + 2ull * a[i] * b[i]; };
  auto lists = [&](uint32_t i) { return a[i] ? (uint64_t)a[i] + b[i] : 0ull; };
  long chunks = 0;
  for (uint32_t n0 = 0; n0 < n; chunks++) {
    const JoinChunk c = join_chunk(a.data(), b.data(), n0, n, lim);
    if (c.end <= n0 || c.end > n) return printf("chunk [%u, %u)\n", n0, c.end), -1;
    uint64_t o = 0, l = 0;
    for (uint32_t i = n0; i < c.end; i++) {
      o += offers(i);
      l += lists(i);
    }
    if (o != c.offers || l != c.lists) return printf("sums at %u\n", n0), -1;
    if (c.end > n0 + 1 && (o > lim.offers || l > lim.lists)) return printf("limit at %u\n", n0), -1;
    if (c.end < n && o + offers(c.end) <= lim.offers && l + lists(c.end) <= lim.lists)
      return printf("short chunk at %u\n", n0), -1;
    n0 = c.end;
  }
  return chunks;
}

int main() {
  long total = 0;
  std::mt19937 rng(5);
  for (int t = 0; t < 200; t++) {
    const uint32_t n = 1 + rng() % 3000;
    std::vector<uint32_t> a(n), b(n);
    for (auto &x : a) x = rng() % 5 ? rng() % 200 : 0;
    for (auto &x : b) x = rng() % 300;
    const long c = check(a, b, JoinLimits{1 + rng() % 2000000, 1 + rng() % 20000});
    if (c < 0) return 1;
    total += c;
  }
  // 20 million nodes of 410 + 600 ids: more list entries than 32 bits count
  const uint32_t n = 20000000;
  std::vector<uint32_t> a(n, 410), b(n, 600);
  const long c = check(a, b, JoinLimits{~0ull, JOIN_LISTS_MAX});
  if (c < 5) return printf("%ld chunks of %u nodes\n", c, n), 1;
  // a wrapped sum would let everything through
  uint32_t wrapped = 0;
  for (uint32_t i = 0; i < n; i++) wrapped += a[i] + b[i];
  if (wrapped == (uint64_t)n * 1010) return printf("the case does not wrap\n"), 1;
  // the descriptors' memory: half of what is free or theirs, not less than
  // they hold or a million, not more than 32 bits count
  const uint64_t G = 1ull << 30;
  if (join_lists_room(100 * G, 0, 16) * 16 > 50 * G || join_lists_room(100 * G, 0, 16) * 16 < 49 * G ||
      join_lists_room(2 * G, 6 * G, 16) * 16 != 6 * G || join_lists_room(10 * G, 2 * G, 16) * 16 != 6 * G ||
      join_lists_room(0, 0, 16) != 1u << 20 || join_lists_room(4096 * G, 0, 16) != JOIN_LISTS_MAX)
    return printf("room for lists\n"), 1;
  printf("OK %ld\n", total + c);
  return 0;
}

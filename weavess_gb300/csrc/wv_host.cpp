#include "wv_host.h"

#include <algorithm>
#include <cstring>

namespace wv {

void GlibcRand::seed_with(uint32_t seed) {
  if (seed == 0) seed = 1;
  int32_t w = (int32_t)seed;
  uint32_t r[34 + 310];
  r[0] = (uint32_t)w;
  for (int k = 1; k < 31; k++) {
    // 16807 * w mod (2^31 - 1) without overflow (Schrage)
    int32_t hi = w / 127773, lo = w % 127773;
    w = 16807 * lo - 2836 * hi;
    if (w < 0) w += 2147483647;
    r[k] = (uint32_t)w;
  }
  for (int k = 31; k < 34; k++) r[k] = r[k - 31];
  for (int k = 34; k < 34 + 310; k++) r[k] = r[k - 31] + r[k - 3];  // discarded outputs
  std::copy(r + 34 + 310 - HIST, r + 34 + 310, w_ + BLOCK);
  pos_ = END;
}

void GlibcRand::refill() {
  std::copy(w_ + BLOCK, w_ + END, w_);
  // the three interleaved chains in registers
  uint32_t a = w_[HIST - 3], b = w_[HIST - 2], c = w_[HIST - 1];
  for (int k = HIST; k < END; k += 3) {
    w_[k] = a += w_[k - 31];
    w_[k + 1] = b += w_[k - 30];
    w_[k + 2] = c += w_[k - 29];
  }
  pos_ = HIST;
}

void gen_random(std::mt19937 &rng, uint32_t *addr, uint32_t size, uint32_t N) {
  for (uint32_t i = 0; i < size; ++i) addr[i] = (uint32_t)(rng() % (N - size));
  std::sort(addr, addr + size);
  for (uint32_t i = 1; i < size; ++i)
    if (addr[i] <= addr[i - 1]) addr[i] = addr[i - 1] + 1;
  uint32_t off = (uint32_t)(rng() % N);
  for (uint32_t i = 0; i < size; ++i) addr[i] = (addr[i] + off) % N;
}

void draw_seeds_rand(RandSource &rnd, uint32_t nq, uint32_t L, uint32_t N, uint32_t *seeds, uint32_t stride) {
  std::vector<uint32_t> sv(nq);
  for (uint32_t q = 0; q < nq; q++) sv[q] = (uint32_t)rnd.next();
#pragma omp parallel for schedule(static)
  for (int64_t q = 0; q < (int64_t)nq; q++) {
    std::mt19937 rng(sv[q]);
    gen_random(rng, seeds + (size_t)q * stride, L, N);
  }
}

namespace {
// small open-addressing id set (ids < 2^32 - 1)
struct IdSet {
  std::vector<uint32_t> slot;
  uint32_t mask;
  explicit IdSet(uint32_t expect) {
    uint32_t cap = 16;
    while (cap < 2 * expect + 2) cap <<= 1;
    slot.assign(cap, 0xffffffffu);
    mask = cap - 1;
  }
  // returns true if inserted (was absent)
  bool insert(uint32_t id) {
    uint32_t h = (id * 2654435761u) & mask;
    while (slot[h] != 0xffffffffu) {
      if (slot[h] == id) return false;
      h = (h + 1) & mask;
    }
    slot[h] = id;
    return true;
  }
};
}  // namespace

void draw_seeds_row(RandSource &rnd, uint32_t L, uint32_t N, const uint32_t *row, uint32_t deg, uint32_t *out) {
  IdSet set(L);
  uint32_t t = 0;
  for (; t < L && t < deg; t++) {
    out[t] = row[t];
    set.insert(row[t]);
  }
  while (t < L) {
    uint32_t id = (uint32_t)rnd.next() % N;
    if (!set.insert(id)) continue;
    out[t++] = id;
  }
}

void draw_seeds_centroid(RandSource &rnd, uint32_t nq, uint32_t L, uint32_t N, const uint32_t *ep_row,
                         uint32_t ep_deg, uint32_t *seeds, uint32_t stride) {
  // draw_seeds_row per query with the taken ids in one bitmap, cleared id by
  // id after each query, where that bitmap has no more words than ids are
  // drawn (setting it up costs less than the draws it serves)
  const uint32_t head = std::min(L, ep_deg);
  const size_t words = ((size_t)N + 63) / 64;
  if (words > (size_t)nq * L || std::any_of(ep_row, ep_row + head, [N](uint32_t id) { return id >= N; })) {
    for (uint32_t q = 0; q < nq; q++) draw_seeds_row(rnd, L, N, ep_row, ep_deg, seeds + (size_t)q * stride);
    return;
  }
  std::vector<uint64_t> bits(words, 0);
  // v % N for v < 2^31: v - floor(v / N) N, the quotient from one product
  const uint64_t inv = ~0ull / N + 1;
  GlibcRand own = rnd.own;  // (a local: its position stays in a register)
  for (uint32_t q = 0; q < nq; q++) {
    uint32_t *out = seeds + (size_t)q * stride;
    uint32_t t = 0;
    for (; t < head; t++) {
      out[t] = ep_row[t];
      bits[ep_row[t] >> 6] |= 1ull << (ep_row[t] & 63);
    }
    while (t < L) {
      const uint32_t v = (uint32_t)(rnd.fn ? rnd.fn() : own.next());
      rnd.drawn++;
      const uint32_t id = N == 1 ? 0u : v - (uint32_t)(((unsigned __int128)inv * v) >> 64) * N;
      uint64_t &w = bits[id >> 6];
      const uint64_t m = 1ull << (id & 63);
      out[t] = id;
      t += (w & m) == 0;
      w |= m;
    }
    for (uint32_t i = 0; i < L; i++) bits[out[i] >> 6] = 0;
  }
  if (!rnd.fn) rnd.own = own;
}

}  // namespace wv

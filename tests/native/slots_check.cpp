// Drives weavess_gb300/csrc/wv_slots.cuh as the InterInsert kernels do (a batch
// of senders' vectors copied ahead, each then refused, appended or taken into a
// re-pruned row) and checks that no slot is taken that is in use or has a copy
// under way.  The same run with slots given back at once must find some.
// Prints "OK <slots taken>" or the first fault.
#include <cstdio>
#include <random>
#include <vector>

#include "../../weavess_gb300/csrc/wv_slots.cuh"

struct Run {
  unsigned spare, R;
  bool at_once;  // the wrong rule: a refused sender's slot is free right away
  wv::Slots s;
  unsigned long long flying = 0, used = 0;  // copies under way; slots of row entries or senders at hand
  std::vector<unsigned> row;
  bool slots_given = false;
  long taken = 0, faults = 0;

  void landed() { flying = 0; }
  unsigned take() {
    const unsigned f = s.take([this]() { landed(); });
    return start(f);
  }
  unsigned start(unsigned f) {
    taken++;
    if (f > R + spare || ((flying | used) >> f & 1)) faults++;
    flying |= 1ull << f;
    used |= 1ull << f;
    return f;
  }
  void drop(unsigned f) {  // a slot whose copy has landed
    s.free |= 1ull << f;
    used &= ~(1ull << f);
  }
  void refuse(int f) {
    if (f < 0) return;
    used &= ~(1ull << f);
    if (at_once) s.free |= 1ull << f;
    else s.give_back((uint32_t)f);
  }
  void insert(std::mt19937 &rng, int fs, unsigned entries) {
    const unsigned what = rng() % 4;
    if (what == 0) return refuse(fs);  // in the row already, or farther than its entries
    if (entries < R && !slots_given) return refuse(fs);
    if (!slots_given) {
      s.reclaim([this]() { landed(); });
      for (unsigned j = 0; j < R; j++) {
        unsigned f = 0;
        while (!(s.free >> f & 1)) f++;
        s.free &= ~(1ull << f);
        row.push_back(start(f));
      }
      slots_given = true;
    }
    const unsigned f = fs < 0 ? take() : (unsigned)fs;
    landed();
    if (row.size() < R) {
      row.push_back(f);
      return;
    }
    if (what == 1) return drop(f);  // occluded
    for (unsigned gone = 1 + rng() % 3; gone && !row.empty(); gone--) {
      const unsigned at = rng() % row.size();
      drop(row[at]);
      row.erase(row.begin() + at);
    }
    row.push_back(f);
  }
  void node(std::mt19937 &rng, unsigned senders) {
    s.reset(R + 1 + spare);
    row.clear();
    used = flying = 0;
    slots_given = false;
    unsigned entries = R - (rng() % 3 == 0 ? rng() % (R < 4 ? R : 4) : 0);
    for (unsigned r0 = 0; r0 < senders;) {
      const unsigned nb = 1 + rng() % 4;
      int fs[4] = {-1, -1, -1, -1};
      for (unsigned k = 0; k < nb; k++)
        if (k < spare && (slots_given || entries == R)) fs[k] = (int)take();
      for (unsigned k = 0; k < nb; k++) {
        insert(rng, fs[k], entries);
        if (!slots_given && entries < R) entries++;
      }
      r0 += nb;
    }
    landed();
  }
};

int main() {
  long taken = 0;
  for (unsigned R : {1u, 2u, 7u, 32u, 59u, 60u, 61u, 62u, 63u}) {
    long wrong = 0;
    for (int at_once = 0; at_once < 2; at_once++) {
      std::mt19937 rng(R);
      Run r{63 - R < 4 ? 63 - R : 4, R, at_once != 0};
      for (int n = 0; n < 2000; n++) r.node(rng, 1 + rng() % 40);
      if (!at_once && r.faults) {
        printf("R=%u: %ld slots taken that were not free\n", R, r.faults);
        return 1;
      }
      taken += at_once ? 0 : r.taken;
      wrong = r.faults;
    }
    if (R < 63 && !wrong) {  // (without spare slots nothing is copied ahead)
      printf("R=%u: the wrong rule went unseen\n", R);
      return 1;
    }
  }
  printf("OK %ld\n", taken);
  return 0;
}

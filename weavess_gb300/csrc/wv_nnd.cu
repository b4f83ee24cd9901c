// K1/K2: INIT_RANDOM and REFINE_NN_DESCENT on GB300.
//
// Replaces ComponentInitRandom::InitInner (src/component_init.cpp:11-45) and
// ComponentRefineNNDescent::RefineInner (src/component_refine.cpp:12-239,
// with nhood::insert / nhood::join, include/weavess/index.h:86-150).
//
// Layout in HBM (n nodes):
//   pool   n x L  {float dist, u32 id|FLAG}  the per-node bounded max-heap, kept
//                 in libstdc++'s heap arrangement between join and update
//   psz, M n      pool sizes, sampled-prefix lengths
//   nnew   n x (S+R), nold n x min(L+R, 2R)  join lists, lnew/lold lengths
//
// The plain form reproduces the single-threaded reference bit for bit:
//  * join: every local-join pair is evaluated (exact-order FP32, or exact
//    integers) and offered both ways ("insert j into i", "insert i into j").
//    Offers that cannot pass nhood::insert's first test (dist > pool max at
//    that time; the max only falls during a join) are dropped at the source;
//    the rest are written grouped by target.  A target's pool after the join
//    is the L least of pool and offers in whatever order they come, except
//    where distances tie: those targets are replayed in the reference's
//    sequential order (keys: node n, pair position in nhood::join, side) by
//    libstdc++'s push_heap/pop_heap, so ties resolve exactly as they do
//    sequentially.  A join whose offers do not fit the device runs in chunks
//    of nodes in node order, all targets replayed, a later chunk seeing the
//    pools the earlier chunks left.
//  * update: per node std::sort (stl_order.cuh), the sampled prefix M, the
//    new/old split and make_heap run as in the reference.  The reverse
//    condition reads pool.back() of the other node as the reference's
//    sequential order sees it: the last slot of its make_heap'd pool if the
//    other node was processed earlier, its maximum otherwise.  Reverse lists
//    are capped at R; each push beyond R overwrites slot rand() % R, the
//    rand() values being drawn on the host, in global (n, l) order, from the
//    context's stream.
//  * the first join is skipped: nhood(L, S) leaves nn_new as 2S zeros
//    (index.h:98-103), which join pairs with nothing.
#include <algorithm>
#include <cstdlib>
#include <string>
#include <vector>

#include "wv_common.cuh"
#include "wv_join_plan.h"
#include "wv_mt.cuh"
#include "wv_nnd.h"
#include "wv_scan.h"

namespace wv {
namespace {

struct Ent {
  float d;
  uint32_t idf;  // id | FLAG when flag (Neighbor::flag) is true
};
struct EntLess {
  __host__ __device__ bool operator()(const Ent &a, const Ent &b) const { return a.d < b.d; }
};

// ---------------------------------------------------------------- mt19937
// std::mt19937 stream of one seed (wv_mt.cuh) by one block.  New word k + 624
// follows from words k, k + 1 and k + 397, so 227 new words depend on old ones
// alone: each step 227 threads make the next 227 words in a ring of 1,024 (the
// words a step writes lie outside those it reads, so one barrier per step).
// Bound by that chain of steps: 1.1 million outputs in 0.5 ms; whole twists in
// place with a barrier on both sides of each part took 0.9 ms.
__global__ void __launch_bounds__(256) k_mt19937(uint32_t seed, uint32_t *out, size_t count) {
  __shared__ uint32_t x[1024];
  const uint32_t t = threadIdx.x;
  if (t == 0) {
    x[0] = seed;
    for (int i = 1; i < 624; i++) x[i] = mt_seed_next(x[i - 1], (uint32_t)i);
  }
  __syncthreads();
  for (size_t b = 0; b < count; b += 227) {
    if (t < 227) {
      const uint32_t k = (uint32_t)(b + t);
      const uint32_t v = mt_mix(x[k & 1023], x[(k + 1) & 1023], x[(k + 397) & 1023]);
      x[(k + 624) & 1023] = v;
      if (b + t < count) out[b + t] = mt_temper(v);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- INIT_RANDOM
// One warp per node: GenRandom from the node's S+1 consecutive mt19937
// outputs, distances (self hits dropped), std::sort of the row.
constexpr int INIT_WARPS = 4;

__global__ void __launch_bounds__(INIT_WARPS * 32)
    k_init_random(const float *__restrict__ base, uint32_t n, uint32_t d, uint32_t S, const uint32_t *__restrict__ mt,
                  uint32_t *ids, float *dist, uint32_t *deg) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t per_warp = (size_t)STAGE_FLOATS * 4 + ((d + 3) & ~3u) * 4 + 64 * sizeof(DI);
  uint8_t *p = smem + warp * per_warp;
  float *stage = (float *)p;
  float *qv = (float *)(p + (size_t)STAGE_FLOATS * 4);
  DI *row = (DI *)(p + (size_t)STAGE_FLOATS * 4 + ((d + 3) & ~3u) * 4);
  const uint32_t gw = gridDim.x * INIT_WARPS;
  for (uint32_t i = blockIdx.x * INIT_WARPS + warp; i < n; i += gw) {
    const uint32_t *r = mt + (size_t)i * (S + 1);
    // addr[j] = rng() % (N - size), sorted (ints: any correct sort agrees)
    uint32_t v = lane < (int)S ? r[lane] % (n - S) : 0xffffffffu;
    for (int k = 2; k <= 32; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        uint32_t o = __shfl_xor_sync(FULL, v, j);
        bool up = (lane & k) == 0, lower = (lane & j) == 0;
        uint32_t lo = min(v, o), hi = max(v, o);
        v = (lower == up) ? lo : hi;
      }
    // bump duplicates: a_j = max(v_j, a_{j-1} + 1) = j + max_{j'<=j}(v_j' - j')
    long long m = (long long)v - lane;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(FULL, m, o);
      if (lane >= o) m = max(m, y);
    }
    uint32_t a = (uint32_t)(m + lane);
    uint32_t off = r[S] % n;
    uint32_t id = (a + off) % n;
    bool keep = lane < (int)S && id != i;
    unsigned km = __ballot_sync(FULL, keep);
    int cnt = __popc(km);
    // compact kept ids (draw order) to lanes 0..cnt-1
    uint32_t *xch = (uint32_t *)row;
    if (keep) xch[__popc(km & ((1u << lane) - 1))] = id;
    for (uint32_t k = lane; k < d; k += 32) qv[k] = base[(size_t)i * d + k];
    __syncwarp();
    uint32_t my = lane < cnt ? xch[lane] : 0u;
    __syncwarp();
    float dd = warp_l2_rows(base, d, my, cnt, qv, stage, lane);
    // std::sort of the row: stable order unless ties with cnt > 16
    float dv = lane < cnt ? dd : __int_as_float(0x7f800000);
    int rank = 0;
    bool tie = false;
    for (int t = 0; t < cnt; t++) {
      float o = __shfl_sync(FULL, dv, t);
      rank += (o < dv) || (o == dv && t < lane);
      tie |= (o == dv && t != lane && lane < cnt);
    }
    tie = __any_sync(FULL, tie);
    if (!tie || cnt <= 16) {
      if (lane < cnt) row[rank] = DI{dd, my};
    } else {
      if (lane < cnt) row[lane] = DI{dd, my};
      __syncwarp();
      if (lane == 0) stl::sort(row, cnt, DILess());
    }
    __syncwarp();
    if (lane < cnt) {
      ids[(size_t)i * S + lane] = row[lane].i;
      dist[(size_t)i * S + lane] = row[lane].d;
    }
    if (lane == 0) deg[i] = cnt;
    __syncwarp();
  }
}

// ---------------------------------------------------------------- INIT_RAND
// ComponentInitRand::InitInner (component_init.cpp:979-1025): node i draws L
// ids by GenRandom from the shared mt19937 stream (outputs [i (L + 1),
// (i + 1)(L + 1))), skips itself, takes the distances (exact reference order,
// a lane per row), and its pool goes through make_heap then std::sort (the
// heap arrangement is where the sort starts, which settles equal
// distances); one warp per node, the two sequential steps on one lane.
constexpr int IR_WARPS = 4;
__host__ __device__ inline size_t init_rand_warp_bytes(uint32_t L, uint32_t d) {
  // a multiple of 16 bytes, so that every warp's query copy starts 16-byte aligned
  const size_t b = (size_t)pow2_ge(L) * 4 + (size_t)L * 4 + (size_t)L * sizeof(DI) + (((size_t)d * 4 + 15) & ~size_t(15));
  return (b + 15) & ~size_t(15);
}
__global__ void __launch_bounds__(IR_WARPS * 32)
    k_init_rand(const float *__restrict__ base, uint32_t n, uint32_t d, uint32_t L, const uint32_t *__restrict__ mt,
                uint32_t *ids, float *dist, uint32_t *deg) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t *p = smem + (size_t)warp * init_rand_warp_bytes(L, d);
  float *qv = reinterpret_cast<float *>(p);
  p += ((size_t)d * 4 + 15) & ~size_t(15);
  DI *pool = reinterpret_cast<DI *>(p);
  p += (size_t)L * sizeof(DI);
  uint32_t *gen = reinterpret_cast<uint32_t *>(p);
  p += (size_t)L * 4;
  uint32_t *key = reinterpret_cast<uint32_t *>(p);
  const unsigned lt = (1u << lane) - 1u;
  for (uint32_t i = blockIdx.x * IR_WARPS + warp; i < n; i += gridDim.x * IR_WARPS) {
    const uint32_t *r = mt + (size_t)i * (L + 1);
    for (uint32_t j = lane; j < L; j += 32) key[j] = r[j] % (n - L);
    for (uint32_t k = lane; k < d; k += 32) qv[k] = base[(size_t)i * d + k];
    __syncwarp();
    warp_gen_random_tail(key, L, r[L] % n, n, gen, lane);
    // the pool in draw order without the node itself
    uint32_t cnt = 0;
    for (uint32_t b = 0; b < L; b += 32) {
      const uint32_t j = b + lane;
      const uint32_t id = j < L ? gen[j] : i;
      const bool keep = j < L && id != i;
      const unsigned km = __ballot_sync(FULL, keep);
      if (keep) {
        const float4 *x = reinterpret_cast<const float4 *>(qv);
        const float4 *y = reinterpret_cast<const float4 *>(base + (size_t)id * d);
        float acc = 0.f;
        for (uint32_t g = 0; g < (d >> 2); g++) acc = __fadd_rn(acc, group4(x[g], __ldg(y + g)));
        pool[cnt + __popc(km & lt)] = DI{acc, id};
      }
      cnt += __popc(km);
    }
    __syncwarp();
    if (lane == 0) {
      stl::make_heap(pool, (int)cnt, DILess());
      stl::sort(pool, (int)cnt, DILess());
    }
    __syncwarp();
    for (uint32_t j = lane; j < cnt; j += 32) {
      ids[(size_t)i * L + j] = pool[j].i;
      dist[(size_t)i * L + j] = pool[j].d;
    }
    if (lane == 0) deg[i] = cnt;
    __syncwarp();
  }
}

// ---------------------------------------------------------------- NN-Descent state
struct Nnd {
  uint32_t n, d, S, K, L, R, capn, capo;
  const float *base;
  const float *xnorm;    // squared row norms (integer data)
  const uint8_t *base8;  // the rows as bytes (integer data, d a multiple of 16 up to 256), or null
  Ent *pool;
  uint32_t *psz, *M;
  uint32_t *nnew, *nold, *lnew, *lold, *pnew, *pold;
  Ent *pre;  // the pools sorted by the last update, flags not yet cleared (n x L; the sampled prefix is M long)
  float *maxd, *hback;
};

// init(): pools <- init rows (flag true), make_heap; M = S.
// efanna: ComponentRefineEFANNA::init (component_refine.cpp:1044-1057) sorts
// the row by distance (std::sort) and skips the node itself and an id equal
// to its predecessor in that order
__global__ void k_nnd_init(Nnd s, const uint32_t *ids, const float *dist, const uint32_t *deg, uint32_t w,
                           int efanna) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  Ent *P = (Ent *)smem + (size_t)threadIdx.x * (s.L + 1);
  if (i >= s.n) return;
  uint32_t sz = min(deg[i], s.L);
  for (uint32_t j = 0; j < sz; j++) P[j] = Ent{dist[(size_t)i * w + j], ids[(size_t)i * w + j] | FLAG};
  if (efanna) {
    stl::sort(P, (int)sz, EntLess());
    uint32_t k = 0, prev = 0;
    for (uint32_t t = 0; t < sz; t++) {
      const uint32_t id = P[t].idf & ID_MASK;
      const bool skip = id == i || (t > 0 && id == prev);
      prev = id;
      if (!skip) P[k++] = P[t];
    }
    sz = k;
    for (uint32_t j = 0; j < sz; j++) s.pre[(size_t)i * s.L + j] = P[j];  // (the first join's sorted pools)
  }
  stl::make_heap(P, (int)sz, EntLess());
  for (uint32_t j = 0; j < sz; j++) s.pool[(size_t)i * s.L + j] = P[j];
  s.psz[i] = sz;
  s.M[i] = s.S;
}

// nhood(L, S, rng, N) (index.h:105-111) for every node: nn_new = GenRandom of
// 2S ids from the shared mt19937 stream (node i reads outputs
// [i (2S + 1), (i + 1)(2S + 1))), nn_old empty.  A warp per node.
constexpr int EF_WARPS = 4;
__global__ void __launch_bounds__(EF_WARPS * 32) k_efanna_nnew(Nnd s, const uint32_t *mtv) {
  extern __shared__ uint32_t ef_key[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t L2 = 2 * s.S;
  uint32_t *key = ef_key + (size_t)warp * pow2_ge(L2);
  for (uint32_t i = blockIdx.x * EF_WARPS + warp; i < s.n; i += gridDim.x * EF_WARPS) {
    const uint32_t *r = mtv + (size_t)i * (L2 + 1);
    for (uint32_t j = lane; j < L2; j += 32) key[j] = r[j] % (s.n - L2);
    __syncwarp();
    warp_gen_random_tail(key, L2, r[L2] % s.n, s.n, s.nnew + (size_t)i * s.capn, lane);
    if (lane == 0) {
      s.lnew[i] = L2;
      s.lold[i] = 0;
    }
  }
}

// update() passes 1-3 for node i: sort, sampled prefix M, new/old lists from
// the pool, flags cleared, make_heap; records the prefix, the sorted maximum
// and the back slot of the heap for the reverse condition.
__global__ void k_upd_sort(Nnd s) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  Ent *P = (Ent *)smem + (size_t)threadIdx.x * (s.L + 1);
  if (i >= s.n) return;
  const uint32_t sz = s.psz[i];
  for (uint32_t j = 0; j < sz; j++) P[j] = s.pool[(size_t)i * s.L + j];
  // a pool the last join left in ascending order (k_apply_fast) is sorted
  bool asc = true;
  for (uint32_t j = 1; j < sz; j++) asc &= P[j - 1].d < P[j].d;
  if (!asc) stl::sort(P, (int)sz, EntLess());
  const uint32_t maxl = min(s.M[i] + s.S, sz);
  uint32_t c = 0, l = 0;
  while (l < maxl && c < s.S) {
    if (P[l].idf & FLAG) ++c;
    ++l;
  }
  s.M[i] = l;
  uint32_t pn = 0, po = 0;
  for (uint32_t j = 0; j < sz; j++) s.pre[(size_t)i * s.L + j] = P[j];
  for (uint32_t j = 0; j < l; j++) {
    uint32_t id = P[j].idf & ID_MASK;
    if (P[j].idf & FLAG) {
      s.nnew[(size_t)i * s.capn + pn++] = id;
    } else {
      // nn_old is truncated to 2R at the end of the update (refine.cpp:231-234)
      if (po < s.capo) s.nold[(size_t)i * s.capo + po] = id;
      po++;
    }
    P[j].idf = id;
  }
  s.pnew[i] = pn;
  s.pold[i] = po;
  s.maxd[i] = sz ? P[sz - 1].d : 0.f;
  stl::make_heap(P, (int)sz, EntLess());
  s.hback[i] = sz ? P[sz - 1].d : 0.f;
  for (uint32_t j = 0; j < sz; j++) s.pool[(size_t)i * s.L + j] = P[j];
}

constexpr int BK_WARPS = 4;
constexpr int BK_CAP = 1024;

// reverse condition of update() pass 3 (component_refine.cpp:191, 202)
__device__ __forceinline__ bool rev_cond(const Nnd &s, uint32_t n, uint32_t o, float dist) {
  float back = o < n ? s.hback[o] : s.maxd[o];
  return dist > back;
}

// events per node and per (target, list) bucket
__global__ void k_upd_count(Nnd s, uint32_t *ecount, uint32_t *bcnt, uint32_t *bmax) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= s.n) return;
  uint32_t cnt = 0;
  for (uint32_t l = 0; l < s.M[n]; l++) {
    Ent e = s.pre[(size_t)n * s.L + l];
    uint32_t o = e.idf & ID_MASK;
    if (rev_cond(s, n, o, e.d)) {
      cnt++;
      uint32_t prev = atomicAdd(&bcnt[2 * o + ((e.idf & FLAG) ? 0 : 1)], 1u);
      if (prev + 1 > BK_CAP) atomicMax(bmax, prev + 1);
    }
  }
  ecount[n] = cnt;
}

__global__ void k_upd_scatter(Nnd s, const uint32_t *eoff, const uint32_t *boff, uint32_t *bcur, uint32_t *bsrc,
                              uint32_t *bflat) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= s.n) return;
  uint32_t f = eoff[n];
  for (uint32_t l = 0; l < s.M[n]; l++) {
    Ent e = s.pre[(size_t)n * s.L + l];
    uint32_t o = e.idf & ID_MASK;
    if (rev_cond(s, n, o, e.d)) {
      uint32_t b = 2 * o + ((e.idf & FLAG) ? 0 : 1);
      uint32_t slot = boff[b] + atomicAdd(&bcur[b], 1u);
      bsrc[slot] = n;
      bflat[slot] = f;
      f++;
    }
  }
}

// sorts one bucket's (src, flat) pairs by src (srcs are distinct) in shared
// memory with a warp bitonic sort; marks events ranked >= R as overflow

__device__ void warp_bitonic_u64(unsigned long long *k, int P, int lane) {
  for (int sz = 2; sz <= P; sz <<= 1)
    for (int j = sz >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < P; i += 32) {
        int l = i ^ j;
        if (l > i) {
          bool up = (i & sz) == 0;
          unsigned long long a = k[i], b = k[l];
          if ((a > b) == up) {
            k[i] = b;
            k[l] = a;
          }
        }
      }
      __syncwarp();
    }
}

__global__ void __launch_bounds__(BK_WARPS * 32)
    k_bucket_sort(uint32_t nb, const uint32_t *boff, const uint32_t *bcnt, uint32_t *bsrc, uint32_t *bflat,
                  uint32_t R, uint32_t *ovf, uint32_t *bigb, uint32_t *nbig) {
  __shared__ unsigned long long keys[BK_WARPS][BK_CAP];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t b = blockIdx.x * BK_WARPS + warp;
  if (b >= nb) return;
  const uint32_t cnt = bcnt[b], off = boff[b];
  if (cnt <= 1) return;
  if (cnt > BK_CAP) {  // left to the block path
    if (lane == 0) bigb[atomicAdd(nbig, 1u)] = b;
    return;
  }
  int P = 1;
  while (P < (int)cnt) P <<= 1;
  unsigned long long *k = keys[warp];
  for (int i = lane; i < P; i += 32)
    k[i] = i < (int)cnt ? ((unsigned long long)bsrc[off + i] << 32) | bflat[off + i] : ~0ull;
  __syncwarp();
  warp_bitonic_u64(k, P, lane);
  for (int i = lane; i < (int)cnt; i += 32) {
    bsrc[off + i] = (uint32_t)(k[i] >> 32);
    bflat[off + i] = (uint32_t)k[i];
    if ((uint32_t)i >= R) ovf[(uint32_t)k[i]] = 1u;
  }
}

// buckets longer than BK_CAP: one block each, bitonic sort in a global
// scratch region of P (power of 2 >= the longest bucket) keys per block
__global__ void __launch_bounds__(1024)
    k_bucket_sort_big(const uint32_t *bigb, const uint32_t *boff, const uint32_t *bcnt, uint32_t *bsrc,
                      uint32_t *bflat, uint32_t R, uint32_t *ovf, unsigned long long *scratch, uint32_t P) {
  const uint32_t b = bigb[blockIdx.x], cnt = bcnt[b], off = boff[b];
  unsigned long long *k = scratch + (size_t)blockIdx.x * P;
  for (uint32_t i = threadIdx.x; i < P; i += blockDim.x)
    k[i] = i < cnt ? ((unsigned long long)bsrc[off + i] << 32) | bflat[off + i] : ~0ull;
  __syncthreads();
  for (uint32_t sz = 2; sz <= P; sz <<= 1)
    for (uint32_t j = sz >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        uint32_t l = i ^ j;
        if (l > i) {
          bool up = (i & sz) == 0;
          unsigned long long x = k[i], y = k[l];
          if ((x > y) == up) {
            k[i] = y;
            k[l] = x;
          }
        }
      }
      __syncthreads();
    }
  for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
    bsrc[off + i] = (uint32_t)(k[i] >> 32);
    bflat[off + i] = (uint32_t)k[i];
    if (i >= R) ovf[(uint32_t)k[i]] = 1u;
  }
}

// update() pass 4: node o's lists = pool part ++ reverse list (first R
// pushes, then the overflow overwrites in order); nn_old truncated to 2R
__global__ void k_bucket_apply(Nnd s, const uint32_t *boff, const uint32_t *bcnt, const uint32_t *bsrc,
                               const uint32_t *bflat, const uint32_t *ovf_ord, const int *rv) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= s.n) return;
  for (int type = 0; type < 2; type++) {
    const uint32_t b = 2 * o + type, cnt = bcnt[b], off = boff[b];
    uint32_t *list = type == 0 ? s.nnew + (size_t)o * s.capn + s.pnew[o] : s.nold + (size_t)o * s.capo + s.pold[o];
    const uint32_t keep = min(cnt, s.R);
    // the part of the reverse list that fits the (truncated) list
    const uint32_t room = type == 0 ? s.capn - s.pnew[o] : (s.pold[o] < 2 * s.R ? 2 * s.R - s.pold[o] : 0u);
    for (uint32_t j = 0; j < keep && j < room; j++) list[j] = bsrc[off + j];
    for (uint32_t j = s.R; j < cnt; j++) {
      uint32_t pos = (uint32_t)rv[ovf_ord[bflat[off + j]]] % s.R;
      if (pos < room) list[pos] = bsrc[off + j];
    }
    if (type == 0) s.lnew[o] = s.pnew[o] + keep;
    else s.lold[o] = min(s.pold[o] + keep, 2 * s.R);
  }
}

// ---------------------------------------------------------------- join
// The local join in two launches.  k_join computes a node's pair distances
// into a dense tile G (rows: new ++ old, columns: new), keeps the offers that
// pass nhood::insert's first test, and writes them grouped by target: the
// entries {distance, candidate} of target p of node n contiguous, one
// descriptor {offset, count, n, p} in the target's own descriptor list.  The
// space of a node's entries is taken with one atomic per node and a
// descriptor's slot with one per (node, target); one atomic per 32 offers on
// a single cursor and one per offer to group them had bound the join.  What
// bounds it now: latency between a node's short phases (lists, rows, tile,
// counts, entries) at 16 warps per SM.  Integer rows come from the byte copy
// (128 bytes a row at d = 128), widened to FP16 once where they are staged
// (not at every fragment, a third of the tile's instructions) and read by
// ldmatrix; the offers are counted and written by a lane per target, without
// a vote per 32 pairs.  The 100k x 128 build (S 10, L 40, R 100) takes
// 29.2 ms, its seven joins 9.9 ms of them; fragments widened on the fly and
// votes cost 2 ms more, and the joins had been 28.6 ms of 82 with the FP32
// rows, the tcgen05 Gram tile and the two atomics.  Six joins of 60k x 96 real-valued (FP32): 18.6 ms with
// those atomics, 14.5 ms without, 13.4 ms with pairs taken two by two, 12.3 ms
// with 32 new rows per tile (the other rows staged half as often).
struct JoinOut {
  uint2 *ent;                  // {distance bits, candidate id}
  uint16_t *eq;                // the candidate's position in the node's list (new ++ old): the replay's key
  unsigned long long *cursor;  // entries asked for (past `cap`: none written, the host retries with room)
  unsigned long long cap;
  uint4 *desc;                 // {offset, count, n, p}, target t's from toff[t]
  const uint32_t *toff;        // prefix sums of the targets' occurrences in the lists
  uint32_t *tcur;              // descriptors written per target
  const float *mx;             // pool maxima (-inf: empty pool)
};
struct JoinCfg {
  uint32_t ti;     // FP32: rows per i tile
  uint32_t tj;     // rows per j tile
  uint32_t gcap;   // floats of G in shared memory; larger tiles take the block's slab of gscr
  float *gscr;
  size_t gslab;
  uint32_t *lscr;  // the node's lists (4 + warps words per entry and block) when they do not fit shared memory
};

constexpr int J_THREADS = 256;
constexpr int J_TI = 16, J_TI_BIG = 32;  // FP32: new rows per i tile (the larger where the tile stays below 64 KB)
constexpr int J_TJ = 64;  // FP32: rows per j tile (new ++ old); fewer for long rows (the tile must fit shared memory)
constexpr int JI_THREADS = 128;       // integer rows
constexpr uint32_t JI_ROWS = 96;      // integer rows staged at once (all of a node's rows, or a 48 x 48 tile)
constexpr uint32_t J_GCAP = 3072;     // floats of G in shared memory

// occurrences of every id in the lists of nodes [n0, n1), a warp per node, the
// largest tile a node needs, and the list entries of all (over 10 million nodes
// of long lists have more than 32 bits count)
__global__ void k_occ_count(Nnd s, uint32_t n0, uint32_t n1, uint32_t *occ, unsigned long long *gmax,
                            unsigned long long *lists) {
  const int lane = threadIdx.x & 31;
  unsigned long long sum = 0;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t n = n0 + w; n < n1; n += nw) {
    const uint32_t a = s.lnew[n], b = s.lold[n];
    if (a == 0) continue;
    const unsigned long long g = (unsigned long long)(a + b) * (a | 1u);
    if (lane == 0 && g > J_GCAP) atomicMax(gmax, g);
    sum += a + b;
    for (uint32_t t = lane; t < a + b; t += 32)
      atomicAdd(&occ[t < a ? s.nnew[(size_t)n * s.capn + t] : s.nold[(size_t)n * s.capo + (t - a)]], 1u);
  }
  if (lane == 0 && sum) atomicAdd(lists, sum);
}

// nhood::insert's first test is against the pool's current maximum, the
// heap's front (an empty pool takes nothing in a join)
__global__ void k_pool_max(Nnd s, float *mx) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < s.n) mx[i] = s.psz[i] > 0 ? s.pool[(size_t)i * s.L].d : __int_as_float(0xff800000);
}

// row stride of integer rows (FP16) in shared memory: an odd multiple of 16
// bytes (ldmatrix then reads eight rows from different banks)
__host__ __device__ inline uint32_t ji_stride(uint32_t d) { return d * 2 + 16; }

// 16 bytes of an integer row as 16 halves: 0x6400 | b is 1024 + b
__device__ __forceinline__ void ji_halves(uint32_t w, uint32_t &lo, uint32_t &hi) {
  const uint32_t k = 0x64646464u, m = 0x64006400u;
  const uint32_t l = __byte_perm(w, k, 0x4140), h = __byte_perm(w, k, 0x4342);
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(lo) : "r"(l), "r"(m));
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(h), "r"(m));
}
__device__ __forceinline__ void ji_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ji_ldm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// distances of rows J (tj of them) x rows I (ti) into G (row j0 + j, column
// i0 + i): dot products of the integer values on the tensor cores (exact in
// FP16; FP32 sums are integers below 2^24 for d <= 256) and the norm form in
// 32-bit integers, converted to the FP32 value the reference's sum gives.
// Rows past ti / tj (in the staging area, whatever it holds) only reach
// columns / rows of the tile that are dropped.
__device__ __forceinline__ void ji_tile(const uint8_t *I, const uint8_t *J, uint32_t stride, uint32_t d, uint32_t ti,
                                        uint32_t tj, uint32_t i0, uint32_t j0, const int *nrm, float *G, uint32_t gs,
                                        int warp, int nwarps, int lane) {
  const int g = lane >> 2, j = lane & 3;
  // ldmatrix: lanes 8 m .. 8 m + 7 give the rows of matrix m.  A: rows 0..7
  // and 8..15 at k, then at k + 8; B: columns 0..7 at k and k + 8, columns
  // 8..15 at k and k + 8
  const uint32_t asm0 = (uint32_t)__cvta_generic_to_shared(J) + (uint32_t)(lane & 15) * stride + (lane >> 4) * 16;
  const uint32_t bsm0 = (uint32_t)__cvta_generic_to_shared(I) + (uint32_t)((lane & 7) + (lane >> 4) * 8) * stride +
                        ((lane >> 3) & 1) * 16;
  for (uint32_t mt = warp; mt * 16 < tj; mt += nwarps) {
    for (uint32_t nb = 0; nb < ti; nb += 32) {
      float acc[4][4];
#pragma unroll
      for (int t = 0; t < 4; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
      const uint32_t as = asm0 + mt * 16 * stride, bs = bsm0 + nb * stride;
      const bool two = nb + 16 < ti;
#pragma unroll 4
      for (uint32_t k = 0; k < d * 2; k += 32) {
        uint32_t a[4], b[4], b2[4];
        ji_ldm(a, as + k);
        ji_ldm(b, bs + k);
        ji_mma(acc[0], a, b[0], b[1]);
        ji_mma(acc[1], a, b[2], b[3]);
        if (two) {
          ji_ldm(b2, bs + 16 * stride + k);
          ji_mma(acc[2], a, b2[0], b2[1]);
          ji_mma(acc[3], a, b2[2], b2[3]);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t jj = mt * 16 + g + h * 8;
        if (jj >= tj) continue;
        const int nj = nrm[j0 + jj];
        float *row = G + (size_t)(j0 + jj) * gs + i0;
#pragma unroll
        for (int t = 0; t < 4; t++) {
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const uint32_t ii = nb + t * 8 + 2 * j + e;
            if (ii < ti) row[ii] = (float)(nj + nrm[i0 + ii] - 2 * __float2int_rn(acc[t][2 * h + e]));
          }
        }
      }
    }
  }
}

// FP32 distances, in the reference's order, of i rows pa, pa + NW (NI of
// them) and this lane's j rows pj, pj + 32 (NJ).  A lane's row is four
// wavefronts of shared memory per 16 bytes, 12 operations of a pair: one pair
// at a time the shared memory bound the join, two by two the arithmetic does.
template <int NI, int NJ>
__device__ __forceinline__ void jf_pairs(const float *ri, const float *rj, uint32_t fs, uint32_t d4, uint32_t pa,
                                         uint32_t nw, uint32_t pj, uint32_t tj, uint32_t i0, uint32_t j0, uint32_t a,
                                         float *G, uint32_t gs) {
  bool need = false;
  auto wanted = [&](int u, int v) {
    const uint32_t gi = i0 + pa + u * nw, gj = j0 + pj + 32 * v;
    return pj + 32 * v < tj && gj > (gj < a ? gi : 0u);
  };
#pragma unroll
  for (int v = 0; v < NJ; v++) need |= wanted(0, v);  // (the first i row wants all the others do)
  if (!need) return;
  const float4 *x[NI], *y[NJ];
#pragma unroll
  for (int u = 0; u < NI; u++) x[u] = reinterpret_cast<const float4 *>(ri + (size_t)(pa + u * nw) * fs);
#pragma unroll
  for (int v = 0; v < NJ; v++) y[v] = reinterpret_cast<const float4 *>(rj + (size_t)min(pj + 32 * v, tj - 1) * fs);
  float dist[NI][NJ];
#pragma unroll
  for (int u = 0; u < NI; u++)
#pragma unroll
    for (int v = 0; v < NJ; v++) dist[u][v] = 0.f;
#pragma unroll 2
  for (uint32_t k = 0; k < d4; k++) {
    float4 xk[NI], yk[NJ];
#pragma unroll
    for (int u = 0; u < NI; u++) xk[u] = x[u][k];
#pragma unroll
    for (int v = 0; v < NJ; v++) yk[v] = y[v][k];
#pragma unroll
    for (int u = 0; u < NI; u++)
#pragma unroll
      for (int v = 0; v < NJ; v++) dist[u][v] = __fadd_rn(dist[u][v], group4(xk[u], yk[v]));
  }
#pragma unroll
  for (int u = 0; u < NI; u++)
#pragma unroll
    for (int v = 0; v < NJ; v++) {
      if (!wanted(u, v)) continue;
      const uint32_t gi = i0 + pa + u * nw, gj = j0 + pj + 32 * v;
      G[(size_t)gj * gs + gi] = dist[u][v];
      if (gj < a) G[(size_t)gi * gs + gj] = dist[u][v];
    }
}

// the local join of nodes [n0, n1), a node per block at a time.  I8: integer
// rows in [0, 255] from the byte copy of the base (d a multiple of 16, d <=
// 256); else FP32 rows, every distance folded in the reference's order.
template <bool I8>
__global__ void __launch_bounds__(I8 ? JI_THREADS : J_THREADS)
    k_join(Nnd s, uint32_t n0, uint32_t n1, JoinOut o, JoinCfg cf, unsigned long long *pairs) {
  constexpr int T = I8 ? JI_THREADS : J_THREADS, NW = T / 32;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ unsigned long long ebase;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t capt = s.capn + s.capo;
  const uint32_t stride = I8 ? ji_stride(s.d) : (((s.d + 3) & ~3u) + 4) * 4;  // bytes
  const size_t rbytes = (size_t)(I8 ? JI_ROWS : cf.ti + cf.tj) * stride;
  float *Gs = reinterpret_cast<float *>(smem + rbytes);
  uint32_t *ids = cf.lscr ? cf.lscr + (size_t)blockIdx.x * (4 + NW) * capt : reinterpret_cast<uint32_t *>(Gs + cf.gcap);
  float *mx = reinterpret_cast<float *>(ids + capt);
  uint32_t *tend = reinterpret_cast<uint32_t *>(mx + capt);  // end of each target's entries
  int *nrm = reinterpret_cast<int *>(tend + capt);           // (I8 only)
  uint32_t *cnt = reinterpret_cast<uint32_t *>(nrm + capt);  // NW x capt
  unsigned long long npairs = 0;
  for (uint32_t n = n0 + blockIdx.x; n < n1; n += gridDim.x) {
    const uint32_t a = s.lnew[n], b = s.lold[n];
    if (a == 0) continue;  // block-uniform
    const uint32_t tot = a + b, gs = a | 1u;
    float *G = (size_t)tot * gs <= cf.gcap ? Gs : cf.gscr + (size_t)blockIdx.x * cf.gslab;
    __syncthreads();  // the previous node's tile and lists are done with
    for (uint32_t t = tid; t < tot; t += T) {
      const uint32_t id = t < a ? s.nnew[(size_t)n * s.capn + t] : s.nold[(size_t)n * s.capo + (t - a)];
      ids[t] = id;
      mx[t] = o.mx[id];
      if (I8) nrm[t] = (int)s.xnorm[id];
    }
    __syncthreads();
    if constexpr (I8) {
      const uint32_t ch = s.d / 16;
      auto stage = [&](uint8_t *dst, uint32_t r0, uint32_t cntr) {
        constexpr int U = 4;  // chunks in flight per thread
        for (uint32_t e0 = tid; e0 < cntr * ch; e0 += U * T) {
          uint4 v[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const uint32_t e = e0 + u * T;
            if (e < cntr * ch)
              v[u] = __ldg(reinterpret_cast<const uint4 *>(s.base8 + (size_t)ids[r0 + e / ch] * s.d) + e % ch);
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            const uint32_t e = e0 + u * T;
            if (e < cntr * ch) {
              uint4 lo, hi;
              ji_halves(v[u].x, lo.x, lo.y);
              ji_halves(v[u].y, lo.z, lo.w);
              ji_halves(v[u].z, hi.x, hi.y);
              ji_halves(v[u].w, hi.z, hi.w);
              uint4 *p = reinterpret_cast<uint4 *>(dst + (size_t)(e / ch) * stride) + 2 * (e % ch);
              p[0] = lo;
              p[1] = hi;
            }
          }
        }
      };
      if (tot <= JI_ROWS) {
        stage(smem, 0, tot);
        __syncthreads();
        ji_tile(smem, smem, stride, s.d, a, tot, 0, 0, nrm, G, gs, warp, NW, lane);
      } else {
        constexpr uint32_t H = JI_ROWS / 2;
        uint8_t *J = smem + (size_t)H * stride;
        for (uint32_t i0 = 0; i0 < a; i0 += H)
          for (uint32_t j0 = 0; j0 < tot; j0 += H) {
            const uint32_t ti = min(H, a - i0), tj = min(H, tot - j0);
            __syncthreads();
            if (j0 == 0) stage(smem, i0, ti);
            stage(J, j0, tj);
            __syncthreads();
            ji_tile(smem, J, stride, s.d, ti, tj, i0, j0, nrm, G, gs, warp, NW, lane);
          }
      }
    } else {
      const uint32_t fs = stride / 4, d4 = s.d >> 2;
      float *ri = reinterpret_cast<float *>(smem);
      float *rj = ri + (size_t)cf.ti * fs;
      for (uint32_t i0 = 0; i0 < a; i0 += cf.ti) {
        const uint32_t ti = min(cf.ti, a - i0);
        for (uint32_t j0 = 0; j0 < tot; j0 += cf.tj) {
          const uint32_t tj = min(cf.tj, tot - j0);
          if (j0 + tj <= min(a, i0 + 1)) continue;  // both new: computed with the roles exchanged
          __syncthreads();
          // stage rows (coalesced 16-byte copies, one row per warp step)
          for (uint32_t r = warp; r < ti + tj; r += NW) {
            const uint32_t id = r < ti ? ids[i0 + r] : ids[j0 + (r - ti)];
            float *dst = r < ti ? ri + (size_t)r * fs : rj + (size_t)(r - ti) * fs;
            const float *src = s.base + (size_t)id * s.d;
            for (uint32_t k = lane; k < d4; k += 32) cp_async16(dst + 4 * k, src + 4 * k);
          }
          cp_async_wait_all();
          __syncthreads();
          // warps take i rows, lanes take j rows; a pair of new rows is
          // computed once (the distance is symmetric bit for bit)
          for (uint32_t pa = warp; pa < ti; pa += 2 * NW) {
            for (uint32_t pj = lane; pj - lane < tj; pj += 64) {
              const bool i2 = pa + NW < ti, j2 = pj - lane + 32 < tj;
              if (i2 && j2) jf_pairs<2, 2>(ri, rj, fs, d4, pa, NW, pj, tj, i0, j0, a, G, gs);
              else if (i2) jf_pairs<2, 1>(ri, rj, fs, d4, pa, NW, pj, tj, i0, j0, a, G, gs);
              else if (j2) jf_pairs<1, 2>(ri, rj, fs, d4, pa, NW, pj, tj, i0, j0, a, G, gs);
              else jf_pairs<1, 1>(ri, rj, fs, d4, pa, NW, pj, tj, i0, j0, a, G, gs);
            }
          }
        }
      }
    }
    __syncthreads();
    // Offers per target: pairs of different ids (a pair of new rows is
    // evaluated in one of its two orders, whatever the positions).  A lane
    // takes a target, a warp every NW-th partner of 32 targets: the tile is
    // read along its rows or columns without conflicts, and nothing is voted
    // on.  cnt[w * capt + p]: warp w's entries for target p, then their ends.
    for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
      const uint32_t p = p0 + lane;
      if (p < tot) {
        const uint32_t pid = ids[p];
        const float m = mx[p];
        uint32_t c = 0, np = 0;
        for (uint32_t q = warp; q < a; q += NW) {
          const uint32_t id = ids[q];
          c += id != pid && G[(size_t)p * gs + q] <= m;
          np += pid < id;
        }
        if (p < a) {
          for (uint32_t q = a + warp; q < tot; q += NW) {
            const bool diff = ids[q] != pid;
            c += diff && G[(size_t)q * gs + p] <= m;
            np += diff;
          }
          npairs += np;
        }
        cnt[warp * capt + p] = c;
      }
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t run = 0;
      for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
        const uint32_t p = p0 + lane;
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) c += p < tot ? cnt[w * capt + p] : 0u;
        uint32_t x = c;
        for (int k = 1; k < 32; k <<= 1) {
          const uint32_t y = __shfl_up_sync(FULL, x, k);
          if (lane >= k) x += y;
        }
        if (p < tot) {
          uint32_t at = run + x - c;  // each warp's first entry of target p
#pragma unroll
          for (int w = 0; w < NW; w++) {
            const uint32_t n1 = cnt[w * capt + p];
            cnt[w * capt + p] = at;
            at += n1;
          }
          tend[p] = at;
        }
        run += __shfl_sync(FULL, x, 31);
      }
      if (lane == 0) ebase = run ? atomicAdd(o.cursor, (unsigned long long)run) : 0ull;
    }
    __syncthreads();
    const uint32_t total = tend[tot - 1];
    if (total == 0 || ebase + total > o.cap) continue;  // block-uniform
    for (uint32_t p = tid; p < tot; p += T) {
      const uint32_t e0 = cnt[p], c = tend[p] - e0;
      if (c) {
        const uint32_t t = ids[p];
        o.desc[o.toff[t] + atomicAdd(&o.tcur[t], 1u)] = make_uint4((uint32_t)(ebase + e0), c, n, p);
      }
    }
    for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
      const uint32_t p = p0 + lane;
      if (p < tot && tend[p] > cnt[p]) {
        const uint32_t pid = ids[p];
        const float m = mx[p];
        size_t at = (size_t)ebase + cnt[warp * capt + p];
        auto put = [&](uint32_t q, uint32_t id, float dist) {
          if (id != pid && dist <= m) {
            o.ent[at] = make_uint2(__float_as_uint(dist), id);
            o.eq[at] = (uint16_t)q;
            at++;
          }
        };
        for (uint32_t q = warp; q < a; q += NW) put(q, ids[q], G[(size_t)p * gs + q]);
        if (p < a)
          for (uint32_t q = a + warp; q < tot; q += NW) put(q, ids[q], G[(size_t)q * gs + p]);
      }
    }
  }
  if (pairs) {
    for (int k = 16; k > 0; k >>= 1) npairs += __shfl_xor_sync(FULL, npairs, k);
    if (lane == 0 && npairs) atomicAdd(pairs, npairs);
  }
}

// ---------------------------------------------------------------- offers into the pools
// A warp reads the entries of one target through up to 32 descriptors at a
// time as one flat range: lane l of step e0 takes entry e0 + l, whose
// descriptor it finds by a binary search over the descriptors' prefix sums.
struct SegBatch {
  uint32_t off, cnt, incl, n, p, total;
  __device__ void load(const uint4 *desc, uint32_t b, uint32_t dn, int lane) {
    const uint4 v = b + lane < dn ? desc[b + lane] : make_uint4(0u, 0u, 0u, 0u);
    off = v.x;
    cnt = v.y;
    n = v.z;
    p = v.w;
    incl = cnt;
    for (int k = 1; k < 32; k <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, k);
      if (lane >= k) incl += y;
    }
    total = __shfl_sync(FULL, incl, 31);
  }
  // the descriptor (lane) of flat entry e < total, and the entry's index
  __device__ int find(uint32_t e, uint32_t &idx) const {
    int lo = 0;
#pragma unroll
    for (int st = 16; st > 0; st >>= 1)
      if (__shfl_sync(FULL, incl, lo + st - 1) <= e) lo += st;
    lo = min(lo, 31);
    const uint32_t ex = __shfl_sync(FULL, incl - cnt, lo);
    idx = __shfl_sync(FULL, off, lo) + (e - ex);
    return lo;
  }
};

// merges up to 32 offers (one per lane, key = distance bits << 32 | id, ~0
// for none) into the sorted pool: repeats of an offer or of a pool entry are
// dropped (the same id has the same distance), the rest are placed by rank.
// fmin: the least distance this lane saw fall off the pool's end.
__device__ __forceinline__ void fast_merge(float *pd, uint32_t *pi, uint32_t &sz, uint32_t L, unsigned long long key, uint32_t *pos,
                           float &fmin, int lane) {
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const unsigned long long y = __shfl_xor_sync(FULL, key, j);
      const bool lower = ((lane & j) == 0) == ((lane & k) == 0);
      key = lower ? (key < y ? key : y) : (key < y ? y : key);
    }
  const unsigned long long prev = __shfl_up_sync(FULL, key, 1);
  bool keep = key != ~0ull && !(lane > 0 && prev == key);
  const float dist = __uint_as_float((uint32_t)(key >> 32));
  const uint32_t id = (uint32_t)key;
  uint32_t lo = 0, hi = keep ? sz : 0u;
  while (lo < hi) {
    const uint32_t m = (lo + hi) >> 1;
    const unsigned long long pk = ((unsigned long long)__float_as_uint(pd[m]) << 32) | (pi[m] & ID_MASK);
    if (pk < key) lo = m + 1;
    else hi = m;
  }
  if (keep && lo < sz && (pi[lo] & ID_MASK) == id && pd[lo] == dist) keep = false;
  const unsigned km = __ballot_sync(FULL, keep);
  if (!km) return;
  const int nk = __popc(km), r = __popc(km & lt);
  if (keep) pos[r] = lo;
  __syncwarp();
  const int first = (int)pos[0];
  for (int jt = (int)sz; jt > first; jt -= 32) {
    const int j = jt - 32 + lane;
    const bool act = j >= first;
    float v = 0.f;
    uint32_t x = 0;
    int np = 0;
    if (act) {
      v = pd[j];
      x = pi[j];
      int l2 = 0, h2 = nk;  // offers placed at or before entry j
      while (l2 < h2) {
        const int m = (l2 + h2) >> 1;
        if ((int)pos[m] <= j) l2 = m + 1;
        else h2 = m;
      }
      np = j + l2;
    }
    __syncwarp();
    if (act) {
      if (np < (int)L) {
        pd[np] = v;
        pi[np] = x;
      } else {
        fmin = fminf(fmin, v);
      }
    }
    __syncwarp();
  }
  if (keep) {
    const uint32_t np = lo + r;
    if (np < L) {
      pd[np] = dist;
      pi[np] = id | FLAG;
    } else {
      fmin = fminf(fmin, dist);
    }
  }
  sz = min(L, sz + (uint32_t)nk);
  __syncwarp();
}

constexpr int AF_WARPS = 8;
constexpr uint32_t AP_WARP_CAP = 1024;   // offers per target for the warp replay
constexpr uint32_t AP_BIG_CAP = 8192;    // offers per target for the block replay in shared memory (power of 2)

// the targets left to the replay, by their number of offers, and the sizes
// the host needs
struct Redo {
  uint32_t *cnt;   // [0] warp, [1] block, [2] block with global scratch, [3] most offers of the last
  uint32_t *list[3];
};
__device__ __forceinline__ void redo_push(const Redo &r, uint32_t t, uint32_t cnt) {
  const int k = cnt <= AP_WARP_CAP ? 0 : cnt <= AP_BIG_CAP ? 1 : 2;
  r.list[k][atomicAdd(r.cnt + k, 1u)] = t;
  if (k == 2) atomicMax(r.cnt + 3, cnt);
}

__host__ __device__ inline size_t af_warp_words(uint32_t L) { return 2 * (((size_t)L + 3) & ~size_t(3)) + 128 + 32; }

// nhood::insert (index.h:120-135) of all of a target's offers, in any order.
// Sequentially an offer enters when it is not farther than the current
// maximum and its id is not pooled, and the maximum leaves a full pool; the
// maximum only falls, so the pool ends as the L least of the pool and the
// offers (repeats once, none above the first maximum).  The heap's
// arrangement depends on the order, but the update that follows sorts the
// pool, so the arrangement matters only where distances tie: a target with
// two equal distances among the kept entries, or between a kept and a dropped
// one, is left as it was and replayed in the reference's order
// (k_replay_*).  Bound by latency (entries from L2, merges in shared memory):
// the seven joins of the 100k x 128 build take 2.1 ms here and 5.2 ms in the
// replays (a tenth of its integer targets tie), against 37 ms when every
// target sorted and replayed its offers; 5.6 + 5.6 ms against 504 ms on the
// six joins of 60k x 96 with up to 100 reverse neighbours.  srt: the pools sorted as the last update left them, flags
// not yet cleared; the first mclr[t] entries' flags are cleared here (null:
// none).
__global__ void __launch_bounds__(AF_WARPS * 32)
    k_apply_fast(Nnd s, const Ent *srt, const uint32_t *mclr, JoinOut o, Redo redo) {
  extern __shared__ __align__(16) uint32_t af_smem[];
  if (*o.cursor > o.cap) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t L = s.L, Lp = (L + 3) & ~3u;
  uint32_t *sm = af_smem + warp * af_warp_words(L);
  float *pd = reinterpret_cast<float *>(sm);
  uint32_t *pi = sm + Lp;
  uint2 *buf = reinterpret_cast<uint2 *>(sm + 2 * Lp);  // 64 waiting offers
  uint32_t *pos = sm + 2 * Lp + 128;
  for (uint32_t t = blockIdx.x * AF_WARPS + warp; t < s.n; t += gridDim.x * AF_WARPS) {
    const uint32_t dn = o.tcur[t];
    if (dn == 0) continue;
    uint32_t sz = s.psz[t];
    const uint32_t mc = mclr ? mclr[t] : 0u;
    for (uint32_t j = lane; j < sz; j += 32) {
      const Ent e = srt[(size_t)t * L + j];
      pd[j] = e.d;
      pi[j] = j < mc ? (e.idf & ID_MASK) : e.idf;
    }
    __syncwarp();
    const float mx0 = pd[sz - 1];  // (a target with offers has a pool)
    float thr = mx0, fmin = __int_as_float(0x7f800000);
    uint32_t nb = 0, offers = 0;
    const uint4 *dsc = o.desc + o.toff[t];
    bool any = false;
    for (uint32_t b = 0; b < dn; b += 32) {
      SegBatch sb;
      sb.load(dsc, b, dn, lane);
      offers += sb.total;
      for (uint32_t e0 = 0; e0 < sb.total; e0 += 64) {
        uint32_t i0, i1;
        sb.find(e0 + lane, i0);
        sb.find(e0 + 32 + lane, i1);
        const bool h0 = e0 + lane < sb.total, h1 = e0 + 32 + lane < sb.total;
        const uint2 v0 = h0 ? __ldg(o.ent + i0) : make_uint2(0u, 0u);
        const uint2 v1 = h1 ? __ldg(o.ent + i1) : make_uint2(0u, 0u);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint2 v = h ? v1 : v0;
          const bool ok = (h ? h1 : h0) && __uint_as_float(v.x) <= thr;
          const unsigned m = __ballot_sync(FULL, ok);
          if (!m) continue;
          if (ok) buf[nb + __popc(m & lt)] = v;
          nb += __popc(m);
          __syncwarp();
          if (nb >= 32) {
            const uint2 w = buf[lane];
            const uint2 rest = lane + 32 < (int)nb ? buf[lane + 32] : make_uint2(0u, 0u);
            __syncwarp();
            buf[lane] = rest;
            nb -= 32;
            __syncwarp();
            fast_merge(pd, pi, sz, L, ((unsigned long long)w.x << 32) | w.y, pos, fmin, lane);
            if (sz == L) thr = pd[L - 1];
            any = true;
          }
        }
      }
    }
    if (nb) {
      const uint2 w = buf[lane];
      fast_merge(pd, pi, sz, L, lane < (int)nb ? ((unsigned long long)w.x << 32) | w.y : ~0ull, pos, fmin, lane);
      any = true;
    }
    if (any) {
      bool tie = sz == L && fmin == pd[L - 1];
      for (uint32_t j = lane; j + 1 < sz; j += 32) tie |= pd[j] == pd[j + 1];
      if (__any_sync(FULL, tie)) {
        if (lane == 0) redo_push(redo, t, offers);
      } else {
        for (uint32_t j = lane; j < sz; j += 32) s.pool[(size_t)t * L + j] = Ent{pd[j], pi[j]};
        if (lane == 0) s.psz[t] = sz;
      }
    }
    __syncwarp();
  }
}

// every target with offers to the replay (joins in several chunks, whose
// heaps must keep the reference's arrangement, and init rows whose distances
// are not those of their ids)
__global__ void k_redo_all(uint32_t n, JoinOut o, Redo redo) {
  if (*o.cursor > o.cap) return;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint32_t dn = o.tcur[t];
  if (!dn) return;
  uint32_t cnt = 0;
  for (uint32_t k = 0; k < dn; k++) cnt += o.desc[o.toff[t] + k].y;
  redo_push(redo, t, cnt);
}

struct WarpSync {
  __device__ void operator()() const { __syncwarp(); }
};
struct BlockSync {
  __device__ void operator()() const { __syncthreads(); }
};

struct Grouped {
  unsigned long long key;
  uint32_t cand;
  float dist;
};

// one warp gathers target t's entries with their keys -- the reference's
// sequential position (node n, pair position in nhood::join's loops, side) --
// into k; batches of 32 descriptors b0, b0 + bstep, ...  `at`: where the
// warp's entries go
__device__ __forceinline__ void gather_offers(const Nnd &s, const JoinOut &o, uint32_t t, uint32_t dn, uint32_t b, uint32_t at,
                              Grouped *k, int lane) {
  SegBatch sb;
  sb.load(o.desc + o.toff[t], b, dn, lane);
  for (uint32_t e0 = 0; e0 < sb.total; e0 += 32) {
    uint32_t idx;
    const int l = sb.find(e0 + lane, idx);
    const uint32_t n = __shfl_sync(FULL, sb.n, l), p = __shfl_sync(FULL, sb.p, l);
    if (e0 + lane < sb.total) {
      const uint2 v = o.ent[idx];
      const uint32_t q = o.eq[idx], a = s.lnew[n], tot = a + s.lold[n];
      // the pair (i, j): i new, and of two new rows the one of smaller id;
      // side 0 offers j to i, side 1 i to j
      const bool side0 = p < a && (q >= a || t < v.y);
      const uint32_t gi = side0 ? p : q, gj = side0 ? q : p;
      k[at + e0 + lane] = Grouped{((unsigned long long)n << 32) | ((gi * tot + gj) << 1) | (side0 ? 0u : 1u), v.y,
                                  __uint_as_float(v.x)};
    }
  }
}

// sorts `cnt` grouped offers by key in shared memory (P = pow2 >= cnt),
// threads [0, nthr) of the calling group cooperate; `sync` orders steps
template <class Sync>
__device__ void bitonic_grouped(Grouped *k, int P, int tid, int nthr, Sync sync) {
  for (int sz = 2; sz <= P; sz <<= 1)
    for (int j = sz >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < P; i += nthr) {
        int l = i ^ j;
        if (l > i) {
          bool up = (i & sz) == 0;
          Grouped a = k[i], b = k[l];
          if ((a.key > b.key) == up) {
            k[i] = b;
            k[l] = a;
          }
        }
      }
      sync();
    }
}

// nhood::insert (index.h:120-135) applied to one target's offers in key order
// by one warp; pool P (heap) in shared memory.  Lane 0 runs the heap steps.
__device__ void apply_offers(Ent *P, uint32_t &sz, uint32_t L, const Grouped *off, uint32_t cnt, int lane) {
  uint32_t i = 0;
  while (i < cnt) {
    const float front = P[0].d;
    const uint32_t j = i + lane;
    bool pass = j < cnt && !(off[j].dist > front);
    unsigned m = __ballot_sync(FULL, pass);
    if (!m) {
      i += 32;
      continue;
    }
    const uint32_t f = i + __ffs(m) - 1;
    const uint32_t cid = off[f].cand;
    bool dup = false;
    for (uint32_t x = lane; x < sz; x += 32) dup |= (P[x].idf & ID_MASK) == cid;
    dup = __any_sync(FULL, dup);
    if (!dup && lane == 0) {
      if (sz < L) {
        P[sz] = Ent{off[f].dist, cid | FLAG};
        sz++;
        stl::push_heap(P, (int)sz, EntLess());
      } else {
        stl::pop_heap(P, (int)sz, EntLess());
        P[sz - 1] = Ent{off[f].dist, cid | FLAG};
        stl::push_heap(P, (int)sz, EntLess());
      }
    }
    sz = __shfl_sync(FULL, sz, 0);
    __syncwarp();
    i = f + 1;
  }
}

// the replay of the targets in redo.list[0]: a warp per target, offers sorted
// by key in shared memory
constexpr int AP_WARPS = 4;
__global__ void __launch_bounds__(AP_WARPS * 32) k_replay_warp(Nnd s, JoinOut o, Redo redo) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Grouped *k = (Grouped *)smem + (size_t)warp * AP_WARP_CAP;
  Ent *P = (Ent *)((Grouped *)smem + (size_t)AP_WARPS * AP_WARP_CAP) + (size_t)warp * (s.L + 1);
  const uint32_t m = redo.cnt[0];
  for (uint32_t w = blockIdx.x * AP_WARPS + warp; w < m; w += gridDim.x * AP_WARPS) {
    const uint32_t t = redo.list[0][w], dn = o.tcur[t];
    uint32_t cnt = 0;
    for (uint32_t b = 0; b < dn; b += 32) {
      uint32_t c = b + lane < dn ? o.desc[o.toff[t] + b + lane].y : 0u;
      for (int x = 16; x > 0; x >>= 1) c += __shfl_xor_sync(FULL, c, x);
      gather_offers(s, o, t, dn, b, cnt, k, lane);
      cnt += c;
    }
    int Pn = 1;
    while (Pn < (int)cnt) Pn <<= 1;
    for (int i = (int)cnt + lane; i < Pn; i += 32) k[i] = Grouped{~0ull, 0u, 0.f};
    uint32_t sz = s.psz[t];
    for (uint32_t i = lane; i < sz; i += 32) P[i] = s.pool[(size_t)t * s.L + i];
    __syncwarp();
    bitonic_grouped(k, Pn, lane, 32, WarpSync());
    apply_offers(P, sz, s.L, k, cnt, lane);
    for (uint32_t i = lane; i < sz; i += 32) s.pool[(size_t)t * s.L + i] = P[i];
    if (lane == 0) s.psz[t] = sz;
    __syncwarp();
  }
}

// the same for the targets of redo.list[1] (offers in shared memory) or
// list[2] (gk: pcap keys of global scratch per block), a block per target
constexpr int AB_THREADS = 512;
__global__ void __launch_bounds__(AB_THREADS) k_replay_block(Nnd s, JoinOut o, Redo redo, Grouped *gk, uint32_t pcap) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Ent *P = (Ent *)smem;
  Grouped *k = gk ? gk + (size_t)blockIdx.x * pcap : (Grouped *)(smem + ((size_t)(s.L + 2) & ~size_t(1)) * sizeof(Ent));
  __shared__ uint32_t szs, fill;
  const int li = gk ? 2 : 1;
  const uint32_t m = redo.cnt[li];
  for (uint32_t w = blockIdx.x; w < m; w += gridDim.x) {
    const uint32_t t = redo.list[li][w], dn = o.tcur[t];
    if (threadIdx.x == 0) fill = 0;
    __syncthreads();
    for (uint32_t b = 32 * warp; b < dn; b += AB_THREADS) {
      uint32_t c = b + lane < dn ? o.desc[o.toff[t] + b + lane].y : 0u, at = 0;
      for (int x = 16; x > 0; x >>= 1) c += __shfl_xor_sync(FULL, c, x);
      if (lane == 0) at = atomicAdd(&fill, c);  // (any order: the keys are sorted next)
      at = __shfl_sync(FULL, at, 0);
      gather_offers(s, o, t, dn, b, at, k, lane);
    }
    __syncthreads();
    const uint32_t cnt = fill;
    int Pn = 1;
    while (Pn < (int)cnt) Pn <<= 1;
    for (int i = (int)cnt + threadIdx.x; i < Pn; i += AB_THREADS) k[i] = Grouped{~0ull, 0u, 0.f};
    const uint32_t sz0 = s.psz[t];
    for (uint32_t i = threadIdx.x; i < sz0; i += AB_THREADS) P[i] = s.pool[(size_t)t * s.L + i];
    __syncthreads();
    bitonic_grouped(k, Pn, threadIdx.x, AB_THREADS, BlockSync());
    if (warp == 0) {
      uint32_t sz = sz0;
      apply_offers(P, sz, s.L, k, cnt, lane);
      if (lane == 0) szs = sz;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < szs; i += AB_THREADS) s.pool[(size_t)t * s.L + i] = P[i];
    if (threadIdx.x == 0) s.psz[t] = szs;
    __syncthreads();
  }
}

// whether every init row's distance is the distance of its ids (the
// reference's order, a lane per entry): *ok = 0 where one is not, and the
// joins then replay every target
__global__ void k_check_rows(Nnd s, const uint32_t *ids, const float *dist, const uint32_t *deg, uint32_t w, int *ok) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5, d4 = s.d >> 2;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < s.n; i += nw) {
    const uint32_t sz = min(deg[i], s.L);
    const float4 *x = reinterpret_cast<const float4 *>(s.base + (size_t)i * s.d);
    for (uint32_t j = lane; j < sz; j += 32) {
      const uint32_t id = ids[(size_t)i * w + j];
      if (id >= s.n) {
        *ok = 0;
        continue;
      }
      const float4 *y = reinterpret_cast<const float4 *>(s.base + (size_t)id * s.d);
      float acc = 0.f;
      for (uint32_t k = 0; k < d4; k++) acc = __fadd_rn(acc, group4(__ldg(x + k), __ldg(y + k)));
      if (__float_as_uint(acc) != __float_as_uint(dist[(size_t)i * w + j])) *ok = 0;
    }
  }
}

// RefineInner tail: sort each pool, keep the first K (PruneNaive)
__global__ void k_nnd_final(Nnd s, uint32_t *ids, float *dist, uint32_t *deg) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  Ent *P = (Ent *)smem + (size_t)threadIdx.x * (s.L + 1);
  if (i >= s.n) return;
  const uint32_t sz = s.psz[i];
  for (uint32_t j = 0; j < sz; j++) P[j] = s.pool[(size_t)i * s.L + j];
  bool asc = true;
  for (uint32_t j = 1; j < sz; j++) asc &= P[j - 1].d < P[j].d;
  if (!asc) stl::sort(P, (int)sz, EntLess());
  const uint32_t k = min(sz, s.K);
  for (uint32_t j = 0; j < k; j++) {
    ids[(size_t)i * s.K + j] = P[j].idf & ID_MASK;
    dist[(size_t)i * s.K + j] = P[j].d;
  }
  deg[i] = k;
}

constexpr int NODE_THREADS = 64;  // threads per block of the per-node sort kernels

}  // namespace

// ================================================================ host side
int mt19937_gpu(wv_ctx *c, uint32_t seed, uint32_t *d_out, size_t count) {
  k_mt19937<<<1, 256, 0, c->stream>>>(seed, d_out, count);
  WV_CUDA(c, cudaGetLastError());
  return WV_OK;
}

int init_random_gpu(wv_ctx *c, uint32_t S) {
  WV_CHECK(c, c->n > 0, WV_ERR_STATE, "no base uploaded");
  WV_CHECK(c, S >= 1 && S <= 32, WV_ERR_LIMIT, "S=%u: this build supports 1 <= S <= 32", S);
  WV_CHECK(c, S < c->n, WV_ERR_ARG, "S=%u must be smaller than n=%u", S, c->n);
  WV_CHECK(c, c->d % 4 == 0, WV_ERR_LIMIT, "dimension %u is not a multiple of 4", c->d);
  cudaError_t e = cudaSuccess;
  const size_t count = (size_t)c->n * (S + 1);
  uint32_t *mt = c->buf<uint32_t>("mt", count, &e);
  WV_CUDA(c, e);
  // `std::mt19937 rng(rand())`: one draw from the process rand() stream
  const uint32_t seed = (uint32_t)c->rnd.next();
  int rc = mt19937_gpu(c, seed, mt, count);
  if (rc) return rc;
  WV_CUDA(c, c->fg_ids.ensure((size_t)c->n * S * 4));
  WV_CUDA(c, c->fg_dist.ensure((size_t)c->n * S * 4));
  WV_CUDA(c, c->fg_deg.ensure((size_t)c->n * 4));
  const size_t smem = INIT_WARPS * ((size_t)STAGE_FLOATS * 4 + ((c->d + 3) & ~3u) * 4 + 64 * sizeof(DI));
  WV_CUDA(c, cudaFuncSetAttribute(k_init_random, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int blocks = (int)std::min<size_t>((c->n + INIT_WARPS - 1) / INIT_WARPS, (size_t)c->sms * 16);
  k_init_random<<<blocks, INIT_WARPS * 32, smem, c->stream>>>(c->base.as<float>(), c->n, c->d, S, mt,
                                                               c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                               c->fg_deg.as<uint32_t>());
  WV_CUDA(c, cudaGetLastError());
  c->fg_n = c->n;
  c->fg_w = S;
  c->fg_has_ep = false;
  c->fg_eps.clear();
  return check_device_status(c, "init_random");
}

int init_rand_gpu(wv_ctx *c, uint32_t L) {
  WV_CHECK(c, c->n > 0, WV_ERR_STATE, "no base uploaded");
  WV_CHECK(c, L >= 1 && L <= 1024, WV_ERR_LIMIT, "L=%u: this build supports 1 <= L <= 1024", L);
  WV_CHECK(c, L < c->n, WV_ERR_ARG, "L=%u must be smaller than n=%u", L, c->n);
  WV_CHECK(c, c->d % 4 == 0, WV_ERR_LIMIT, "dimension %u is not a multiple of 4", c->d);
  cudaError_t e = cudaSuccess;
  const size_t count = (size_t)c->n * (L + 1);
  uint32_t *mt = c->buf<uint32_t>("mt", count, &e);
  WV_CUDA(c, e);
  // `std::mt19937 rng(rand())`: one draw from the process rand() stream
  const uint32_t seed = (uint32_t)c->rnd.next();
  int rc = mt19937_gpu(c, seed, mt, count);
  if (rc) return rc;
  WV_CUDA(c, c->fg_ids.ensure((size_t)c->n * L * 4));
  WV_CUDA(c, c->fg_dist.ensure((size_t)c->n * L * 4));
  WV_CUDA(c, c->fg_deg.ensure((size_t)c->n * 4));
  const size_t smem = IR_WARPS * init_rand_warp_bytes(L, c->d);
  WV_CHECK(c, smem <= 227 * 1024, WV_ERR_LIMIT, "L=%u d=%u need %zu bytes of shared memory", L, c->d, smem);
  WV_CUDA(c, cudaFuncSetAttribute(k_init_rand, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int blocks = (int)std::min<size_t>((c->n + IR_WARPS - 1) / IR_WARPS, (size_t)c->sms * 16);
  k_init_rand<<<blocks, IR_WARPS * 32, smem, c->stream>>>(c->base.as<float>(), c->n, c->d, L, mt,
                                                           c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                           c->fg_deg.as<uint32_t>());
  WV_CUDA(c, cudaGetLastError());
  c->fg_n = c->n;
  c->fg_w = L;
  c->fg_has_ep = false;
  c->fg_eps.clear();
  return check_device_status(c, "init_rand");
}

int nndescent_gpu(wv_ctx *c, const NndParams &p, NndStats *st) {
  WV_CHECK(c, c->n > 0 && c->fg_n == c->n, WV_ERR_STATE, "NN-Descent needs the base and an initial graph");
  WV_CHECK(c, p.L >= 1 && p.K >= 1 && p.S >= 1 && p.R >= 1, WV_ERR_ARG, "S, K, L, R must be positive");
  WV_CHECK(c, p.L <= 256, WV_ERR_LIMIT, "L=%u above the supported 256", p.L);
  WV_CHECK(c, c->d % 4 == 0, WV_ERR_LIMIT, "dimension %u is not a multiple of 4", c->d);
  // the join key packs (pair position << 1 | side) into 32 bits
  WV_CHECK(c, 2ull * (p.S + p.R) * (p.S + 3ull * p.R) < (1ull << 31), WV_ERR_LIMIT, "S=%u R=%u too large", p.S, p.R);
  NndStats local;
  NndStats &S = st ? *st : local;
  S = NndStats();
  cudaError_t e = cudaSuccess;
  const uint32_t n = c->n;
  Nnd s{};
  s.n = n;
  s.d = c->d;
  s.S = p.S;
  s.K = p.K;
  s.L = p.L;
  s.R = p.R;
  s.capn = std::max(p.S + p.R, 2 * p.S);  // EFANNA's first nn_new holds 2S ids
  s.capo = std::min(p.L + p.R, 2 * p.R);
  s.base = c->base.as<float>();
  s.xnorm = c->base_int ? c->xnorm.as<float>() : nullptr;
  s.base8 = c->base_int && c->base8.p ? c->base8.as<uint8_t>() : nullptr;
  s.pool = c->buf<Ent>("pool", (size_t)n * p.L, &e);
  s.psz = c->buf<uint32_t>("psz", n, &e);
  s.M = c->buf<uint32_t>("M", n, &e);
  s.nnew = c->buf<uint32_t>("nnew", (size_t)n * s.capn, &e);
  s.nold = c->buf<uint32_t>("nold", (size_t)n * s.capo, &e);
  s.lnew = c->buf<uint32_t>("lnew", n, &e);
  s.lold = c->buf<uint32_t>("lold", n, &e);
  s.pnew = c->buf<uint32_t>("pnew", n, &e);
  s.pold = c->buf<uint32_t>("pold", n, &e);
  s.pre = c->buf<Ent>("pre", (size_t)n * p.L, &e);
  s.maxd = c->buf<float>("maxd", n, &e);
  s.hback = c->buf<float>("hback", n, &e);
  uint32_t *ecount = c->buf<uint32_t>("ecount", n, &e);
  uint32_t *eoff = c->buf<uint32_t>("eoff", n + 1, &e);
  uint32_t *bcnt = c->buf<uint32_t>("bcnt", 2 * (size_t)n, &e);
  uint32_t *boff = c->buf<uint32_t>("boff", 2 * (size_t)n + 1, &e);
  uint32_t *bcur = c->buf<uint32_t>("bcur", 2 * (size_t)n, &e);
  uint32_t *scan_tmp = c->buf<uint32_t>("scan", scan_scratch_words((size_t)n * p.L + 2 * (size_t)n), &e);
  uint32_t *tcnt = c->buf<uint32_t>("tcnt", n, &e);
  uint32_t *toff = c->buf<uint32_t>("toff", n + 1, &e);
  uint32_t *tcur = c->buf<uint32_t>("tcur", n, &e);
  uint32_t *act = c->buf<uint32_t>("act", n, &e);
  uint32_t *big = c->buf<uint32_t>("big", n, &e);
  uint32_t *small = c->buf<uint32_t>("small", 16, &e);  // [0] nact [1] nbig [2] maxseg [3] cursor
  uint32_t *usmall = c->buf<uint32_t>("usmall", 8, &e);  // [0] longest big bucket [1] big buckets
  uint32_t *bigb = c->buf<uint32_t>("bigb", 2 * (size_t)n, &e);
  unsigned long long *pairs = (unsigned long long *)c->buf<uint64_t>("pairs", 2, &e);
  WV_CUDA(c, e);

  // The entry buffers hold a whole join's offers: they start at 64 per node
  // and grow to what a join asks for while the device has room for twice
  // that; otherwise (or with WV_NND_OFFER_CAP, which caps them) the join runs
  // in chunks of nodes in node order whose offers' upper bound fits.  Results
  // do not depend on it.
  uint64_t cap_max = ~0ull;
  if (const char *env = getenv("WV_NND_OFFER_CAP")) cap_max = std::max<uint64_t>(1024u, (uint64_t)atol(env));
  uint64_t cap = 0;
  JoinOut jo{};
  auto room = [&](uint64_t want) -> int {  // entry buffers for `want` offers (0: as many as there is memory for)
    want = std::min<uint64_t>(want, std::min<uint64_t>(cap_max, 0xfffffff0ull));
    if (want <= cap) return WV_OK;
    size_t free_b = 0, total_b = 0;
    WV_CUDA(c, cudaMemGetInfo(&free_b, &total_b));
    const uint64_t have = free_b + c->work["of_e"].bytes + c->work["of_q"].bytes;
    want = std::min<uint64_t>(want, std::max<uint64_t>(have / 2 / 10, 1u << 20));
    if (want <= cap) return WV_OK;
    cudaError_t e2 = cudaSuccess;
    jo.ent = c->buf<uint2>("of_e", want, &e2);
    jo.eq = c->buf<uint16_t>("of_q", want, &e2);
    WV_CUDA(c, e2);
    cap = std::min<uint64_t>(c->work["of_e"].bytes / sizeof(uint2), c->work["of_q"].bytes / sizeof(uint16_t));
    cap = std::min<uint64_t>(cap, std::min<uint64_t>(cap_max, 0xfffffff0ull));
    jo.cap = cap;
    return WV_OK;
  };
  {
    const int rc = room((uint64_t)n * 64);
    if (rc) return rc;
  }
  jo.cursor = reinterpret_cast<unsigned long long *>(small);
  jo.toff = toff;
  jo.tcur = tcur;
  float *pmax = c->buf<float>("pmax", n, &e);
  Redo redo{};
  redo.cnt = small + 2;
  redo.list[0] = act;
  redo.list[1] = big;
  redo.list[2] = c->buf<uint32_t>("act2", n, &e);
  WV_CUDA(c, e);
  jo.mx = pmax;

  cudaEvent_t ev0, ev1;
  cudaEventCreate(&ev0);
  cudaEventCreate(&ev1);

  const int nb = (int)((n + NODE_THREADS - 1) / NODE_THREADS);
  const size_t node_smem = (size_t)NODE_THREADS * (p.L + 1) * sizeof(Ent);
  WV_CUDA(c, cudaFuncSetAttribute(k_nnd_init, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)node_smem));
  WV_CUDA(c, cudaFuncSetAttribute(k_upd_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)node_smem));
  WV_CUDA(c, cudaFuncSetAttribute(k_nnd_final, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)node_smem));
  if (p.efanna) {
    // one rand() seeds the mt19937 the nhoods draw their first nn_new from
    WV_CHECK(c, 2ull * p.S < n, WV_ERR_ARG, "EFANNA needs 2S < n (S=%u, n=%u)", p.S, n);
    std::vector<uint32_t> hdeg(n);
    WV_CUDA(c, cudaMemcpyAsync(hdeg.data(), c->fg_deg.p, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    for (uint32_t i = 0; i < n; i++)
      WV_CHECK(c, hdeg[i] <= p.L, WV_ERR_LIMIT, "init row %u has %u entries > L=%u (the pool would outgrow L)", i,
               hdeg[i], p.L);
    const uint32_t seed = (uint32_t)c->rnd.next();
    const size_t count = (size_t)n * (2 * p.S + 1);
    uint32_t *mtv = c->buf<uint32_t>("ef_mt", count, &e);
    WV_CUDA(c, e);
    int rc = mt19937_gpu(c, seed, mtv, count);
    if (rc) return rc;
    const size_t ef_smem = (size_t)EF_WARPS * pow2_ge(2 * p.S) * 4;
    WV_CUDA(c, cudaFuncSetAttribute(k_efanna_nnew, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ef_smem));
    k_efanna_nnew<<<c->sms * 8, EF_WARPS * 32, ef_smem, c->stream>>>(s, mtv);
    WV_CUDA(c, cudaGetLastError());
  }
  k_nnd_init<<<nb, NODE_THREADS, node_smem, c->stream>>>(s, c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                          c->fg_deg.as<uint32_t>(), c->fg_w, p.efanna ? 1 : 0);
  WV_CUDA(c, cudaGetLastError());

  // the local join's pair distances: from the byte rows on the tensor cores
  // for integer data with d a multiple of 16 up to 256 (WV_NND_JOIN=fp32
  // keeps the FP32 kernel), else in FP32 in the reference's order.  Both give
  // the same offers.
  const char *join_env = getenv("WV_NND_JOIN");
  const bool join_i8 = c->base_int && s.base8 && !(join_env && std::string(join_env) == "fp32");
  const uint32_t capt = s.capn + s.capo;
  JoinCfg jc{};
  jc.tj = J_TJ;
  jc.gcap = J_GCAP;
  // shared memory: the rows, then the tile and the node's lists as far as
  // they fit (else they live in global memory, a slab per block)
  const uint32_t fstride = ((c->d + 3) & ~3u) + 4;
  jc.ti = (size_t)(J_TI_BIG + J_TJ) * fstride * 4 <= 64 * 1024 ? J_TI_BIG : J_TI;
  if (!join_i8)
    while (jc.tj > 32 && (size_t)(jc.ti + jc.tj) * fstride * 4 > 200 * 1024) jc.tj -= 32;
  size_t join_smem = join_i8 ? (size_t)JI_ROWS * ji_stride(c->d) : (size_t)(jc.ti + jc.tj) * fstride * 4;
  const uint32_t lwords = 4 + (join_i8 ? JI_THREADS : J_THREADS) / 32;  // words per list entry
  const size_t lists = (size_t)capt * lwords * 4;
  const bool lists_smem = join_smem + lists <= 200 * 1024;
  if (lists_smem) join_smem += lists;
  if (join_smem + (size_t)jc.gcap * 4 <= 220 * 1024) join_smem += (size_t)jc.gcap * 4;
  else jc.gcap = 0;
  WV_CHECK(c, join_smem + 16 <= 227 * 1024, WV_ERR_LIMIT, "dimension %u too large for the local-join tile", c->d);
  int jper = 0;
  if (join_i8) {
    WV_CUDA(c, cudaFuncSetAttribute(k_join<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)join_smem));
    WV_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&jper, k_join<true>, JI_THREADS, join_smem));
  } else {
    WV_CUDA(c, cudaFuncSetAttribute(k_join<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)join_smem));
    WV_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&jper, k_join<false>, J_THREADS, join_smem));
  }
  WV_CHECK(c, jper > 0, WV_ERR_LIMIT, "the local join does not fit the device (d=%u)", c->d);
  const uint32_t jgrid = (uint32_t)(c->sms * jper);
  if (!lists_smem) jc.lscr = c->buf<uint32_t>("join_l", (size_t)jgrid * lwords * capt, &e);
  WV_CUDA(c, e);
  const size_t af_smem = AF_WARPS * af_warp_words(p.L) * 4;
  WV_CUDA(c, cudaFuncSetAttribute(k_apply_fast, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)af_smem));
  const size_t apw_smem = (size_t)AP_WARPS * AP_WARP_CAP * sizeof(Grouped) + (size_t)AP_WARPS * (p.L + 1) * sizeof(Ent);
  WV_CUDA(c, cudaFuncSetAttribute(k_replay_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)apw_smem));
  const size_t apb_pool = ((size_t)(p.L + 2) & ~size_t(1)) * sizeof(Ent);
  const size_t apb_smem = (size_t)AP_BIG_CAP * sizeof(Grouped) + apb_pool;
  WV_CUDA(c, cudaFuncSetAttribute(k_replay_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)apb_smem));
  WV_CUDA(c, cudaMemsetAsync(pairs, 0, 8, c->stream));

  // the init rows' distances must be those of their ids for the order-free
  // application of the offers (k_apply_fast)
  bool dist_ok = true;
  {
    int *ok = reinterpret_cast<int *>(usmall + 4);
    WV_CUDA(c, cudaMemsetAsync(ok, 1, 4, c->stream));
    k_check_rows<<<c->sms * 8, 256, 0, c->stream>>>(s, c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                    c->fg_deg.as<uint32_t>(), c->fg_w, ok);
    WV_CUDA(c, cudaGetLastError());
    int h = 0;
    WV_CUDA(c, cudaMemcpyAsync(&h, ok, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    dist_ok = h != 0;
  }

  // list entries per launch: what their descriptors may take of the device's
  // memory beside the entry buffers, asked where they have to grow
  // (WV_NND_LIST_CAP caps them further)
  uint64_t lists_cap = JOIN_LISTS_MAX, lists_max = 0;
  if (const char *env = getenv("WV_NND_LIST_CAP"))
    lists_cap = std::min<uint64_t>(lists_cap, std::max<uint64_t>(1024u, (uint64_t)atol(env)));
  auto lists_room = [&](uint64_t want) -> int {
    const uint64_t held = c->work["of_d"].bytes;
    lists_max = std::min<uint64_t>(lists_cap, held / sizeof(uint4));
    if (want < lists_max) return WV_OK;
    size_t free_b = 0, total_b = 0;
    WV_CUDA(c, cudaMemGetInfo(&free_b, &total_b));
    lists_max = std::min(lists_cap, join_lists_room(free_b, held, sizeof(uint4)));
    return WV_OK;
  };

  // one join over nodes [n0, n1); `whole`: all nodes at once.  Nothing is
  // applied when its lists exceed the limit (fits = false) or its offers the
  // entry buffers (hs.cursor > cap).
  bool fits = true;
  struct {
    unsigned long long cursor;
    uint32_t redo[4];
  } hs;
  auto join = [&](uint32_t n0, uint32_t n1, bool whole, const uint32_t *mclr) -> int {
    WV_CUDA(c, cudaMemsetAsync(tcnt, 0, (size_t)n * 4, c->stream));
    const int ob = (int)std::min<uint32_t>((n1 - n0 + 7) / 8, (uint32_t)c->sms * 16);
    unsigned long long *gmax = reinterpret_cast<unsigned long long *>(small) + 4, hc[2];  // largest tile, list entries
    WV_CUDA(c, cudaMemsetAsync(small, 0, 48, c->stream));
    k_occ_count<<<ob, 256, 0, c->stream>>>(s, n0, n1, tcnt, gmax, gmax + 1);
    WV_CUDA(c, exclusive_scan_u32(tcnt, toff, n, scan_tmp, c->stream));
    WV_CUDA(c, cudaMemsetAsync(tcur, 0, (size_t)n * 4, c->stream));
    WV_CUDA(c, cudaMemcpyAsync(hc, gmax, 16, cudaMemcpyDeviceToHost, c->stream));
    k_pool_max<<<nb, NODE_THREADS, 0, c->stream>>>(s, pmax);
    WV_CUDA(c, cudaGetLastError());
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    unsigned long long hg = hc[0];
    if (whole) {
      const int rl = lists_room(hc[1]);
      if (rl) return rl;
      fits = hc[1] <= lists_max;
      if (!fits) return WV_OK;
    }
    cudaError_t e2 = cudaSuccess;  // (of the buffers sized below)
    jo.desc = c->buf<uint4>("of_d", (size_t)hc[1], &e2);
    WV_CUDA(c, e2);
    uint32_t grid = std::min(jgrid, n1 - n0);
    if (jc.gcap == 0) hg = std::max<unsigned long long>(hg, J_GCAP);
    if (hg > jc.gcap) {  // some tiles live in global memory
      size_t free_b = 0, total_b = 0;
      WV_CUDA(c, cudaMemGetInfo(&free_b, &total_b));
      jc.gslab = (size_t)hg;
      grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(grid, (free_b + c->work["join_g"].bytes) / 4 / (hg * 4)));
      jc.gscr = c->buf<float>("join_g", (size_t)grid * jc.gslab, &e2);
      WV_CUDA(c, e2);
    }
    if (join_i8) k_join<true><<<grid, JI_THREADS, join_smem, c->stream>>>(s, n0, n1, jo, jc, pairs + 1);
    else k_join<false><<<grid, J_THREADS, join_smem, c->stream>>>(s, n0, n1, jo, jc, pairs + 1);
    WV_CUDA(c, cudaGetLastError());
    if (whole && dist_ok)
      k_apply_fast<<<(int)std::min<uint32_t>((n + AF_WARPS - 1) / AF_WARPS, (uint32_t)c->sms * 16), AF_WARPS * 32,
                     af_smem, c->stream>>>(s, s.pre, mclr, jo, redo);
    else
      k_redo_all<<<nb, NODE_THREADS, 0, c->stream>>>(n, jo, redo);
    k_replay_warp<<<c->sms * 3, AP_WARPS * 32, apw_smem, c->stream>>>(s, jo, redo);
    k_replay_block<<<c->sms, AB_THREADS, apb_smem, c->stream>>>(s, jo, redo, nullptr, 0);
    WV_CUDA(c, cudaGetLastError());
    WV_CUDA(c, cudaMemcpyAsync(&hs, small, sizeof(hs), cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    if (hs.redo[2]) {  // targets whose offers exceed shared memory
      uint32_t P = 1;
      while (P < hs.redo[3]) P <<= 1;
      const uint32_t blocks = std::min<uint32_t>(hs.redo[2], (uint32_t)c->sms);
      Grouped *gk = c->buf<Grouped>("of_g", (size_t)blocks * P, &e2);
      WV_CUDA(c, e2);
      k_replay_block<<<blocks, AB_THREADS, apb_pool, c->stream>>>(s, jo, redo, gk, P);
      WV_CUDA(c, cudaGetLastError());
    }
    return WV_OK;
  };
  // the pairs of a retried join count once
  auto take_pairs = [&](bool keep) -> int {
    unsigned long long h = 0;
    if (keep) {
      WV_CUDA(c, cudaMemcpyAsync(&h, pairs + 1, 8, cudaMemcpyDeviceToHost, c->stream));
      WV_CUDA(c, cudaStreamSynchronize(c->stream));
      S.pairs += h;
    }
    WV_CUDA(c, cudaMemsetAsync(pairs + 1, 0, 8, c->stream));
    return WV_OK;
  };
  {
    const int rc = take_pairs(false);
    if (rc) return rc;
  }
  bool chunked = false;  // joins no longer fit in one piece
  for (uint32_t it = 0; it < p.ITER; it++) {
    // ------------------------------------------------------------ join
    // (NN_DESCENT's first join pairs 2S zero ids -- nothing; EFANNA's is live)
    if (it > 0 || p.efanna) {
      cudaEventRecord(ev0, c->stream);
      const uint32_t *mclr = it > 0 ? s.M : nullptr;
      bool done = false;
      while (!chunked && !done) {
        int rc = join(0, n, true, mclr);
        if (rc) return rc;
        if (!fits) {
          chunked = true;
          break;
        }
        if (hs.cursor <= cap) {
          done = true;
          S.offers += hs.cursor;
          S.chunks++;
          rc = take_pairs(true);
          if (rc) return rc;
          break;
        }
        rc = take_pairs(false);
        if (rc) return rc;
        const uint64_t old = cap;
        rc = room(hs.cursor + hs.cursor / 8);
        if (rc) return rc;
        if (cap < hs.cursor || cap == old) chunked = true;
      }
      if (!done) {
        std::vector<uint32_t> h_lnew(n), h_lold(n);
        WV_CUDA(c, cudaMemcpyAsync(h_lnew.data(), s.lnew, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
        WV_CUDA(c, cudaMemcpyAsync(h_lold.data(), s.lold, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
        WV_CUDA(c, cudaStreamSynchronize(c->stream));
        uint32_t n0 = 0;
        while (n0 < n) {
          int rc = lists_room(JOIN_LISTS_MAX);
          if (rc) return rc;
          const JoinChunk ch = join_chunk(h_lnew.data(), h_lold.data(), n0, n, JoinLimits{cap, lists_max});
          const uint32_t n1 = ch.end;
          WV_CHECK(c, ch.offers <= cap, WV_ERR_LIMIT, "node %u alone may produce %llu offers (> %llu)", n0,
                   (unsigned long long)ch.offers, (unsigned long long)cap);
          WV_CHECK(c, ch.lists <= lists_max, WV_ERR_LIMIT, "node %u alone lists %llu ids (> %llu)", n0,
                   (unsigned long long)ch.lists, (unsigned long long)lists_max);
          rc = join(n0, n1, false, nullptr);
          if (rc) return rc;
          WV_CHECK(c, hs.cursor <= cap, WV_ERR_STATE, "a join chunk produced more offers than its bound");
          S.offers += hs.cursor;
          S.chunks++;
          rc = take_pairs(true);
          if (rc) return rc;
          n0 = n1;
        }
      }
      cudaEventRecord(ev1, c->stream);
      cudaEventSynchronize(ev1);
      float ms = 0;
      cudaEventElapsedTime(&ms, ev0, ev1);
      S.ms_join += ms;
    }
    // ------------------------------------------------------------ update
    cudaEventRecord(ev0, c->stream);
    k_upd_sort<<<nb, NODE_THREADS, node_smem, c->stream>>>(s);
    WV_CUDA(c, cudaMemsetAsync(bcnt, 0, 2 * (size_t)n * 4, c->stream));
    WV_CUDA(c, cudaMemsetAsync(usmall, 0, 8, c->stream));
    k_upd_count<<<nb, NODE_THREADS, 0, c->stream>>>(s, ecount, bcnt, usmall);
    WV_CUDA(c, exclusive_scan_u32(ecount, eoff, n, scan_tmp, c->stream));
    WV_CUDA(c, exclusive_scan_u32(bcnt, boff, 2 * (size_t)n, scan_tmp, c->stream));
    uint32_t tail[2];
    WV_CUDA(c, cudaMemcpyAsync(&tail[0], eoff + n - 1, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaMemcpyAsync(&tail[1], ecount + n - 1, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    const uint32_t E = tail[0] + tail[1];
    uint32_t *bsrc = c->buf<uint32_t>("bsrc", E + 1, &e);
    uint32_t *bflat = c->buf<uint32_t>("bflat", E + 1, &e);
    uint32_t *ovf = c->buf<uint32_t>("ovf", E + 1, &e);
    uint32_t *ovf_ord = c->buf<uint32_t>("ovf_ord", E + 1, &e);
    uint32_t *scan_e = c->buf<uint32_t>("scan_e", scan_scratch_words(E + 1), &e);
    WV_CUDA(c, e);
    WV_CUDA(c, cudaMemsetAsync(bcur, 0, 2 * (size_t)n * 4, c->stream));
    WV_CUDA(c, cudaMemsetAsync(ovf, 0, (size_t)(E + 1) * 4, c->stream));
    k_upd_scatter<<<nb, NODE_THREADS, 0, c->stream>>>(s, eoff, boff, bcur, bsrc, bflat);
    const uint32_t nbk = 2 * n;
    k_bucket_sort<<<(nbk + BK_WARPS - 1) / BK_WARPS, BK_WARPS * 32, 0, c->stream>>>(nbk, boff, bcnt, bsrc, bflat,
                                                                                    p.R, ovf, bigb, usmall + 1);
    WV_CUDA(c, cudaGetLastError());
    uint32_t hb[2];
    WV_CUDA(c, cudaMemcpyAsync(hb, usmall, 8, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    if (hb[1]) {
      uint32_t P = 1;
      while (P < hb[0]) P <<= 1;
      unsigned long long *bscr = c->buf<unsigned long long>("bscr", (size_t)hb[1] * P, &e);
      WV_CUDA(c, e);
      k_bucket_sort_big<<<hb[1], 1024, 0, c->stream>>>(bigb, boff, bcnt, bsrc, bflat, p.R, ovf, bscr, P);
      WV_CUDA(c, cudaGetLastError());
    }
    WV_CUDA(c, exclusive_scan_u32(ovf, ovf_ord, (size_t)E + 1, scan_e, c->stream));
    uint32_t nov = 0;
    WV_CUDA(c, cudaMemcpyAsync(&nov, ovf_ord + E, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    int rc = check_device_status(c, "nndescent update");
    if (rc) return rc;
    // the overflow overwrites consume rand() in (n, l) order
    std::vector<int> hrv(nov + 1);
    for (uint32_t k = 0; k < nov; k++) hrv[k] = c->rnd.next();
    int *rv = c->buf<int>("rv", nov + 1, &e);
    WV_CUDA(c, e);
    WV_CUDA(c, cudaMemcpyAsync(rv, hrv.data(), (size_t)(nov + 1) * 4, cudaMemcpyHostToDevice, c->stream));
    k_bucket_apply<<<nb, NODE_THREADS, 0, c->stream>>>(s, boff, bcnt, bsrc, bflat, ovf_ord, rv);
    WV_CUDA(c, cudaGetLastError());
    S.overflow_events += nov;
    cudaEventRecord(ev1, c->stream);
    WV_CUDA(c, cudaEventSynchronize(ev1));
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0, ev1);
    S.ms_update += ms;
  }
  // ------------------------------------------------------------ tail
  WV_CUDA(c, c->fg_ids.ensure((size_t)n * p.K * 4));
  WV_CUDA(c, c->fg_dist.ensure((size_t)n * p.K * 4));
  WV_CUDA(c, c->fg_deg.ensure((size_t)n * 4));
  k_nnd_final<<<nb, NODE_THREADS, node_smem, c->stream>>>(s, c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                           c->fg_deg.as<uint32_t>());
  WV_CUDA(c, cudaGetLastError());
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  c->fg_w = p.K;
  c->fg_has_ep = false;
  c->fg_eps.clear();
  return check_device_status(c, "nndescent");
}

}  // namespace wv

// K3/K4/K5: the Vamana, NSG and SSG link (REFINE_VAMANA / REFINE_NSG /
// REFINE_SSG) on GB300.
//
// Replaces ComponentRefineVAMANA::RefineInner / Link / InterInsert
// (src/component_refine.cpp:794-950), ComponentRefineNSG::RefineInner / Link /
// InterInsert (component_refine.cpp:393-541), ComponentRefineSSG::
// RefineInner / Link / InterInsert (component_refine.cpp:550-720),
// ComponentCandidateNSG and ComponentCandidatePropagation2
// (component_candidate.cpp:10-109), ComponentPruneVAMANA / ComponentPruneNSG /
// ComponentPruneSSG (component_prune.cpp:20-122, 245-300) and
// ComponentRefineEntryCentroid (component_entry.cpp:9-92).
// ComponentConnNSGDFS finds what the entry reaches on the GPU, walks the other
// nodes on the host (the depth-first walk fixes which nodes get linked) and
// batches its greedy searches on the GPU, taken in repair order; ComponentConnSSGDFS (component_conn.cpp:
// 169-225) walks on the GPU (frontier kernels) with the repairs on the device.
//
// Plain form, bit-exact with the single-threaded reference:
//  * candidates: the beam kernel in build mode (seeds flagged, every visit
//    recorded in order), seeds drawn on the host in node order;
//  * prune: a block per node sorts the visit pool by (distance, id) and walks
//    it 128 candidates at a time; nodes where the order of equal distances
//    could matter are redone in the order of std::sort (warp_sort.cuh).
//    VAMANA refills from the skipped items as libstdc++'s heap pops them;
//  * InterInsert: sequentially, node n walks its current row and inserts
//    itself into each neighbour's row (dedup, append, or re-prune).  Node n's
//    row at that moment is its pruned row plus the insertions from nodes < n
//    that still listed n -- and those can only be nodes m < n with n in m's
//    PRUNED row.  So nodes run in id order across all warps, each waiting for
//    those lower ids' rows and applying their insertions in id order, which
//    gives its row at its turn (kept as a snapshot).  Then every row applies,
//    in id order, the insertions from higher ids, read from their snapshots.
//    Each warp keeps its row's vectors and their pairwise distances in shared
//    memory, so an insertion costs one new distance column.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <string>
#include <type_traits>
#include <vector>

#include "warp_sort.cuh"
#include "wv_bfs.cuh"
#include "wv_colsum.cuh"
#include "wv_common.cuh"
#include "wv_link.h"
#include "wv_scan.h"
#include "wv_search.h"
#include "wv_segsort.h"
#include "wv_slots.cuh"

namespace wv {
namespace {

constexpr uint32_t LINK_MAX_R = 63;  // row slots (R + 1) index a 64-bit mask

// exact-order squared L2 of two base rows, read from global memory by one lane
__device__ __forceinline__ float l2g(const float *__restrict__ base, uint32_t d, uint32_t a, uint32_t b) {
  const float4 *x = reinterpret_cast<const float4 *>(base + (size_t)a * d);
  const float4 *y = reinterpret_cast<const float4 *>(base + (size_t)b * d);
  float acc = 0.f;
  const uint32_t d4 = d >> 2;
#pragma unroll 4
  for (uint32_t g = 0; g < d4; g++) acc = __fadd_rn(acc, group4(__ldg(x + g), __ldg(y + g)));
  return acc;
}

struct HeapItem {  // Index::MinHeap<float, SimpleNeighbor>::Item
  float key;
  DI data;
};
struct HeapItemLess {  // Item::operator< is key > other.key
  __device__ bool operator()(const HeapItem &a, const HeapItem &b) const { return a.key > b.key; }
};

// ---------------------------------------------------------------- prune
struct PruneArgs {
  const float *base;
  uint32_t d, n;
  DI *vis;              // chunk x vcap pools (sorted in place)
  const uint32_t *vcnt;
  uint32_t vcap;
  uint32_t n0, cnt;     // nodes [n0, n0 + cnt)
  uint32_t R;
  float alpha;
  uint32_t maxc;        // NSG: C_refine
  float threshold;      // SSG: cos of the angle bound
  const uint32_t *g_ids;  // NSG: the candidate graph (final_graph_)
  const uint32_t *g_deg;
  uint32_t gw;
  int clean;            // Vamana: a short pool is sorted too (clean mode)
  const float *xnorm;   // integer rows: their squared norms
  int *gscr;            // per block: 2 * vcap + 256 ints (EXACT, pools beyond shared memory)
  HeapItem *hscr;       // per block: vcap items (EXACT VAMANA refill)
  uint32_t *out_ids;    // rows of width R, indexed by node
  float *out_dist;
  uint32_t *out_deg;
  int *status;
};

// the angle test of ComponentPruneSSG / RefineSSG::InterInsert
// (component_prune.cpp:96-104, component_refine.cpp:685-693) with the
// reference's operand types: float sums, a float quotient by 2, and the
// quotient by ::sqrt(double) of the float product taken in double, then
// stored to float
__device__ __forceinline__ bool ssg_occludes(float pd, float rd, float djk, float threshold) {
  const float num = __fmul_rn(__fsub_rn(__fadd_rn(pd, rd), djk), 0.5f);  // x / 2 is exact as x * 0.5
  const double den = __dsqrt_rn((double)__fmul_rn(pd, rd));
  const float cos_ij = __double2float_rn(__ddiv_rn((double)num, den));
  return cos_ij > threshold;
}

// ---- the prune with a block per node
// The walk over a node's sorted pool needs its order only where distances
// differ: the pool is sorted by (distance, id), and a node where equal
// distances could have come out in another order is left to the EXACT form,
// which sorts as std::sort does -- two picks of equal distance, a candidate
// occluded by a pick of its own distance, equal distances on both sides of
// the examination bound, or among the entries a Vamana refill takes.  Pools
// of more than 1,024 entries are sorted a window at a time, as far as the
// walk gets.  A
// candidate is tested against the picks until one occludes it: a warp takes
// 32 candidates, drops the occluded ones after each test and, once 16 (8) are
// left, tests them against two (four) picks at a time; the survivors of the
// block's four warps are then picked in order, each pick tested against the
// rest.  On integer data the rows are bytes and the distances exact integers
// (__dp4a), else FP32 sums in the reference's order.
//
// What bounds it: latency of the short phases and barriers; a block's rows,
// picks and sort keys take 34 KB (d = 128 bytes), so 6 nodes per SM are in
// flight.  A warp per node with every pool sorted by the introsort replica in
// global memory and all pairs of a batch as Gram tiles (29 KB per warp, 4
// warps per SM) took 193 ms for the NSG prune of 200k x 128 nodes; this takes
// 17 ms and the EXACT redo 2.8 ms.  Two real-valued Vamana prunes of 20k x 96
// (pools of 1,800 and 4,400): 33 ms -> 13.3 ms.
constexpr int PF_THREADS = 128, PF_NW = PF_THREADS / 32, PF_SIZES = 4;
// pool sizes of the launches
__host__ __device__ constexpr uint32_t pf_keys(int l) { return 1024u << l; }

struct PruneFast {
  const uint8_t *base8;   // byte rows (I8)
  uint32_t keys;          // longest pool this launch takes (a pf_keys value)
  uint32_t cs;            // bytes of a row in shared memory (0: rows read where they lie)
  const uint32_t *list, *nlist;  // the pools (null: all)
  uint32_t *more, *nmore;  // longer pools, for the next launch (null: to redo)
  uint32_t *redo, *nredo;  // pools for the EXACT launch
};

constexpr uint32_t PF_WINDOW = 1024;  // keys sorted at a time
constexpr uint32_t PF_SAVED = 128;    // skipped keys of the first window kept for the Vamana refill
__host__ __device__ inline size_t pf_smem(uint32_t keys, uint32_t cs, uint32_t R, bool exact) {
  return (size_t)keys * 8 + (keys > PF_WINDOW && !exact ? PF_WINDOW * 8 : 0) + PF_WINDOW / 8 + PF_SAVED * 8 +
         (size_t)cs * (32 * PF_NW + R + 1) + (exact ? (2 * (size_t)keys + 256) * 4 : 0);
}

template <int E>
__device__ __noinline__ void pf_sort(unsigned long long *K) {
  constexpr int N = PF_THREADS * E;
  const int tid = threadIdx.x;
  unsigned long long v[E];
#pragma unroll
  for (int e = 0; e < E; e++) v[e] = K[e * PF_THREADS + tid];  // (any assignment: the sort starts here)
  auto cx = [](unsigned long long &a, unsigned long long &b, bool up) {
    const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
    a = up ? lo : hi;
    b = up ? hi : lo;
  };
  // element tid * E + e in v[e]; sizes up to E inside a thread
#pragma unroll
  for (int k = 2; k <= E; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int e = 0; e < E; e++)
        if ((e & j) == 0) cx(v[e], v[e | j], k < E ? (e & k) == 0 : (tid & 1) == 0);
  for (int k = 2 * E; k <= N; k <<= 1) {
    const bool up = ((tid * E) & k) == 0;
    for (int j = k >> 1; j >= E; j >>= 1) {
      const int tm = j / E;
      const bool keep_lo = ((tid & tm) == 0) == up;
      if (tm >= 32) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) K[e * PF_THREADS + tid] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) {
          const unsigned long long o = K[e * PF_THREADS + (tid ^ tm)];
          v[e] = keep_lo ? (v[e] < o ? v[e] : o) : (v[e] < o ? o : v[e]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; e++) {
          const unsigned long long o = __shfl_xor_sync(FULL, v[e], tm);
          v[e] = keep_lo ? (v[e] < o ? v[e] : o) : (v[e] < o ? o : v[e]);
        }
      }
    }
#pragma unroll
    for (int j = E >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int e = 0; e < E; e++)
        if ((e & j) == 0) cx(v[e], v[e | j], up);
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < E; e++) K[tid * E + e] = v[e];
  __syncthreads();
}

// the next keys of a long pool: those above `lo` (the last window's end) up
// to a distance that PF_WINDOW of them do not exceed, unsorted into W (padded
// with ~0).  A linear histogram over the remaining keys' distance bits finds
// it; keys of one distance share a bin, so no window ends between equal
// distances.  Returns the keys taken (0: a bin alone exceeds the window) and
// the new bound in lo.  hist: PF_WINDOW words, W itself.
__device__ __noinline__ uint32_t pf_window(const unsigned long long *U, uint32_t m, unsigned long long *W,
                                           uint32_t &lo, bool first) {
  __shared__ uint32_t mn, mx, bin, taken;
  uint32_t *hist = reinterpret_cast<uint32_t *>(W);
  const int tid = threadIdx.x;
  // (distances are below 2^31 as bits; bits >= lo remain)
  if (tid == 0) {
    mn = 0xffffffffu;
    mx = 0;
    taken = 0;
    bin = 0;
  }
  for (uint32_t i = tid; i < PF_WINDOW; i += PF_THREADS) hist[i] = 0;
  __syncthreads();
  const uint32_t from = first ? 0u : lo;
  uint32_t a = 0xffffffffu, b = 0;
  for (uint32_t i = tid; i < m; i += PF_THREADS) {
    const uint32_t d = (uint32_t)(U[i] >> 32);
    if (d >= from) {
      a = min(a, d);
      b = max(b, d);
    }
  }
  a = __reduce_min_sync(FULL, a);
  b = __reduce_max_sync(FULL, b);
  if ((tid & 31) == 0) {
    atomicMin(&mn, a);
    atomicMax(&mx, b);
  }
  __syncthreads();
  const uint32_t base = mn;
  if (base > mx) return 0;  // (nothing left; block-uniform)
  uint32_t sh = 0;
  while (((mx - base) >> sh) >= PF_WINDOW) sh++;
  for (uint32_t i = tid; i < m; i += PF_THREADS) {
    const uint32_t d = (uint32_t)(U[i] >> 32);
    if (d >= from) atomicAdd(&hist[(d - base) >> sh], 1u);
  }
  __syncthreads();
  if (tid < 32) {  // bins that fit, from the nearest
    uint32_t run = 0, nb = 0;
    for (uint32_t b0 = 0; b0 < PF_WINDOW; b0 += 32) {
      const uint32_t c = hist[b0 + tid];
      uint32_t x = c;
      for (int k = 1; k < 32; k <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, k);
        if (tid >= k) x += y;
      }
      const unsigned over = __ballot_sync(FULL, run + x > PF_WINDOW);
      if (over) {
        nb = b0 + __ffs(over) - 1;
        break;
      }
      run += __shfl_sync(FULL, x, 31);
      nb = b0 + 32;
    }
    if (tid == 0) bin = nb;
  }
  __syncthreads();
  const uint32_t nb = bin;
  if (nb == 0) return 0;
  for (uint32_t i = tid; i < PF_WINDOW; i += PF_THREADS) W[i] = ~0ull;
  __syncthreads();
  for (uint32_t i = tid; i < m; i += PF_THREADS) {
    const unsigned long long k = U[i];
    const uint32_t d = (uint32_t)(k >> 32);
    if (d >= from && ((d - base) >> sh) < nb) W[atomicAdd(&taken, 1u)] = k;
  }
  __syncthreads();
  // the first distance of bin nb (past the last bin: above every distance)
  const unsigned long long next = (unsigned long long)base + ((unsigned long long)nb << sh);
  lo = next > 0xffffffffull ? 0xffffffffu : (uint32_t)next;
  return taken;
}

// distance of two rows: bytes (with their squared norms), or FP32 in the
// reference's order
template <bool I8>
__device__ __forceinline__ float pf_dist(const uint8_t *x, const uint8_t *y, uint32_t d, int nx, int ny) {
  if (I8) {
    unsigned dot = 0, dot2 = 0;
    const uint4 *p = reinterpret_cast<const uint4 *>(x), *q = reinterpret_cast<const uint4 *>(y);
#pragma unroll 4
    for (uint32_t k = 0; k < d / 16; k++) {
      const uint4 u = p[k], v = q[k];
      dot = __dp4a(u.x, v.x, dot);
      dot2 = __dp4a(u.y, v.y, dot2);
      dot = __dp4a(u.z, v.z, dot);
      dot2 = __dp4a(u.w, v.w, dot2);
    }
    return (float)(nx + ny - 2 * (int)(dot + dot2));
  }
  const float4 *p = reinterpret_cast<const float4 *>(x), *q = reinterpret_cast<const float4 *>(y);
  float acc = 0.f;
#pragma unroll 4
  for (uint32_t k = 0; k < d / 4; k++) acc = __fadd_rn(acc, group4(p[k], q[k]));
  return acc;
}

// MODE: 0 Vamana, 1 NSG, 2 SSG.  EXACT: the pools in f.list in std::sort's
// order (warp_sort.cuh; in shared memory up to f.keys entries, else in place)
// and the Vamana refill through libstdc++'s heap steps.
template <int MODE, bool I8, bool EXACT>
__global__ void __launch_bounds__(PF_THREADS) k_prune_block(PruneArgs a, PruneFast f) {
  constexpr bool NSG = MODE != 0;
  extern __shared__ __align__(16) uint8_t pf_sm[];
  __shared__ float pd[LINK_MAX_R];
  __shared__ uint32_t pid[LINK_MAX_R];
  __shared__ int pnrm[LINK_MAX_R];
  __shared__ uint32_t wl[PF_NW][32], wc[PF_NW];
  __shared__ int amb;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  // U: the pool's keys; K: the sorted window (U itself when one window holds
  // every pool)
  unsigned long long *U = reinterpret_cast<unsigned long long *>(pf_sm);
  const bool windows = !EXACT && f.keys > PF_WINDOW;
  unsigned long long *K = windows ? U + f.keys : U;
  unsigned long long *saved = U + f.keys + (windows ? PF_WINDOW : 0u);
  uint32_t *gone = reinterpret_cast<uint32_t *>(saved + PF_SAVED);  // picked or dropped, by position in the window
  uint8_t *cand = reinterpret_cast<uint8_t *>(gone) + PF_WINDOW / 8;  // 32 rows per warp
  uint8_t *pick = cand + (size_t)f.cs * 32 * PF_NW;                           // R rows
  uint8_t *self = pick + (size_t)f.cs * a.R;
  int *scr = reinterpret_cast<int *>(self + f.cs);  // (EXACT)
  HeapItem *heap = EXACT ? a.hscr + (size_t)blockIdx.x * a.vcap : nullptr;
  const uint32_t rb = I8 ? a.d : a.d * 4, d = a.d;
  const uint8_t *rows = I8 ? f.base8 : reinterpret_cast<const uint8_t *>(a.base);
  const bool cv = !NSG && a.clean;
  const uint32_t count = f.nlist ? *f.nlist : a.cnt;
  auto occludes = [&](float cd, float qd, float dd) {
    return MODE == 2 ? ssg_occludes(cd, qd, dd, a.threshold) : (NSG ? (dd < cd) : (__fmul_rn(a.alpha, dd) < cd));
  };
  for (uint32_t it = blockIdx.x; it < count; it += gridDim.x) {
    const uint32_t qi = f.list ? f.list[it] : it, node = a.n0 + qi;
    DI *pool = a.vis + (size_t)qi * a.vcap;
    const uint32_t mv = min(a.vcnt[qi], a.vcap);
    uint32_t *oid = a.out_ids + (size_t)node * a.R;
    float *od = a.out_dist + (size_t)node * a.R;
    const uint32_t deg = (NSG || cv) ? min(a.g_deg[node], a.gw) : 0u;
    if (mv + deg > a.vcap && tid == 0) set_err(a.status, DEV_OVERFLOW);
    const uint32_t m = min(mv + deg, a.vcap);
    if (!NSG && m <= a.R && !a.clean) {  // PruneVAMANA keeps a short pool unsorted
      for (uint32_t j = tid; j < m; j += PF_THREADS) {
        oid[j] = pool[j].i;
        od[j] = pool[j].d;
      }
      if (tid == 0) a.out_deg[node] = m;
      continue;
    }
    if (m == 0) {
      if (tid == 0) a.out_deg[node] = 0;
      continue;
    }
    if (!EXACT && m > f.keys) {
      if (tid == 0) {
        if (f.more) f.more[atomicAdd(f.nmore, 1u)] = qi;
        else f.redo[atomicAdd(f.nredo, 1u)] = qi;
      }
      continue;
    }
    __syncthreads();  // the previous node's shared memory is done with
    if (tid == 0) amb = 0;
    const uint8_t *srow = rows + (size_t)node * rb;
    if (f.cs && deg) {
      for (uint32_t k = tid; k < rb / 16; k += PF_THREADS)
        reinterpret_cast<uint4 *>(self)[k] = __ldg(reinterpret_cast<const uint4 *>(srow) + k);
      srow = self;
    }
    DI *P = m <= f.keys ? reinterpret_cast<DI *>(K) : pool;  // (EXACT)
    const uint32_t N = windows ? m : PF_WINDOW;
    bool bad = false;
    if (EXACT) {
      if (P != pool)
        for (uint32_t i = tid; i < mv; i += PF_THREADS) P[i] = pool[i];
    }
    for (uint32_t i = tid; !EXACT && i < N; i += PF_THREADS) {
      unsigned long long key = ~0ull;
      if (i < mv) {
        const DI x = pool[i];
        key = ((unsigned long long)__float_as_uint(x.d) << 32) | x.i;
        bad |= __float_as_uint(x.d) > 0x7f800000u;  // (negative or NaN: not ordered by its bits)
      }
      if (i < mv || i >= m) U[i] = key;
    }
    __syncthreads();
    // the node's own row joins the pool, distances recomputed
    // (component_prune.cpp:26-34); vcap leaves room for it
    for (uint32_t j = tid; j < m - mv; j += PF_THREADS) {
      uint32_t id = a.g_ids[(size_t)node * a.gw + j];
      if (id >= a.n) {
        set_err(a.status, DEV_BAD_ID);
        id = 0;
      }
      const float x = pf_dist<I8>(srow, rows + (size_t)id * rb, d, I8 ? (int)__ldg(a.xnorm + node) : 0,
                                  I8 ? (int)__ldg(a.xnorm + id) : 0);
      if (EXACT) {
        P[mv + j] = DI{x, id};
      } else {
        U[mv + j] = ((unsigned long long)__float_as_uint(x) << 32) | id;
        bad |= __float_as_uint(x) > 0x7f800000u;
      }
    }
    if (bad) amb = 1;
    __syncthreads();
    if (!EXACT && amb) {  // block-uniform
      if (tid == 0) f.redo[atomicAdd(f.nredo, 1u)] = qi;
      continue;
    }
    if (EXACT) {
      if (warp == 0) {
        int *sc = P != pool ? scr : a.gscr + (size_t)blockIdx.x * (2 * (size_t)a.vcap + 256);
        const uint32_t cap = P != pool ? f.keys : a.vcap;
        warp_std_sort(P, (int)m, DILess(), WarpSortScratch{sc, sc + cap, sc + 2 * cap, sc + 2 * cap + 192}, lane);
      }
      __syncthreads();
    }
    // the window [w0g, w0g + wn) of the sorted pool in K
    uint32_t wn = m, wlo = 0;
    if (!EXACT) {
      if (windows) {
        wn = pf_window(U, m, K, wlo, true);
        if (wn == 0) {  // block-uniform
          if (tid == 0) f.redo[atomicAdd(f.nredo, 1u)] = qi;
          continue;
        }
      }
      pf_sort<PF_WINDOW / PF_THREADS>(K);
    }
    auto kd = [&](uint32_t i) { return EXACT ? P[i].d : __uint_as_float((uint32_t)(K[i] >> 32)); };
    auto ki = [&](uint32_t i) { return EXACT ? P[i].i : (uint32_t)K[i]; };
    // row of sorted entry i into the pick area (a warp)
    auto put_pick = [&](uint32_t slot, const uint8_t *src) {
      for (uint32_t k = lane; k < rb / 16; k += 32)
        reinterpret_cast<uint4 *>(pick + (size_t)slot * f.cs)[k] = reinterpret_cast<const uint4 *>(src)[k];
    };
    uint32_t np = 0, ex = 0, end = m, nskip = 0;
    if (NSG) {
      // start skips the node itself at position 0; pool[start] is taken as is
      const uint32_t start = ki(0) == node ? 1u : 0u;
      if (start >= wn) {
        if (tid == 0) {
          if (start >= m) a.out_deg[node] = 0;
          else f.redo[atomicAdd(f.nredo, 1u)] = qi;  // (the first window ends before it)
        }
        continue;
      }
      if (tid == 0) {
        if (start)
          for (uint32_t i = 1; i < wn && kd(i) == kd(0); i++)
            if (ki(i) != node) amb = 1;  // whether the node comes first depends on the sort
        if (a.R == 1 && start + 1 < wn && kd(start + 1) == kd(start)) amb = 1;
        pid[0] = ki(start);
        pd[0] = kd(start);
        if (I8) pnrm[0] = (int)__ldg(a.xnorm + ki(start));
      }
      if (f.cs && warp == 0) put_pick(0, rows + (size_t)ki(start) * rb);
      np = 1;
      ex = start + 1;
      end = MODE == 2 ? m : min(m, a.maxc);  // SSG examines the whole pool
    }
    __syncthreads();
    bool done = np >= a.R;
    uint32_t wbase = 0, nsaved = 0;  // pool position of the window; keys in `saved`
    bool all_saved = true;
    while (true) {  // windows
    const uint32_t wend = min(wn, end - wbase);
    if (!EXACT) {
      for (uint32_t i = tid; i < PF_WINDOW / 32; i += PF_THREADS) gone[i] = 0;
      __syncthreads();
    }
    while (!done && ex < wend) {
      const uint32_t g0 = EXACT ? ex : 0u;  // position of gone's first bit
      if (EXACT) {
        if (tid < PF_NW) gone[tid] = 0;
        __syncthreads();
      }
      const uint32_t w0 = ex + 32 * warp;
      const uint32_t wcnt = w0 < wend ? min(32u, wend - w0) : 0u;
      float cd = 0.f;
      uint32_t cid = 0;
      int cn = 0;
      if (lane < wcnt) {
        cd = kd(w0 + lane);
        cid = ki(w0 + lane);
        if (I8) cn = (int)__ldg(a.xnorm + cid);
      }
      uint8_t *wrow = cand + (size_t)f.cs * 32 * warp;
      if (f.cs) {
        const uint32_t ch = rb / 16;
        for (uint32_t e = lane; e < ch * 32; e += 32) {  // (warp-uniform trips: e / ch is any row)
          const uint32_t r = e / ch, k = e % ch;
          const uint32_t id = __shfl_sync(FULL, cid, r);
          if (r < wcnt) cp_async16(wrow + (size_t)r * f.cs + k * 16, rows + (size_t)id * rb + k * 16);
        }
        cp_async_wait_all();
        __syncwarp();
      }
      auto row_of = [&](uint32_t c, uint32_t id) { return f.cs ? wrow + (size_t)c * f.cs : rows + (size_t)id * rb; };
      auto pick_row = [&](uint32_t p) { return f.cs ? pick + (size_t)p * f.cs : rows + (size_t)pid[p] * rb; };
      // drops candidate c (bit of the sorted position): clean Vamana's node
      // itself and ids picked before
      auto drop = [&](uint32_t c) { atomicOr(&gone[(w0 - g0 + c) >> 5], 1u << ((w0 - g0 + c) & 31)); };
      // the candidates against the picks so far; wl[warp]: those left, in order
      bool self_hit = cv && lane < wcnt && cid == node;
      if (self_hit) drop(lane);
      unsigned am = __ballot_sync(FULL, lane < wcnt && !self_hit);
      uint32_t A = __popc(am);
      if ((am >> lane) & 1u) wl[warp][__popc(am & lt)] = lane;
      __syncwarp();
      for (uint32_t j = 0; j < np && A > 0;) {
        const uint32_t W = A <= 8 ? 8u : A <= 16 ? 16u : 32u, G = 32 / W;
        const uint32_t at = lane & (W - 1), p = j + lane / W;
        const bool on = at < A && p < np;
        const uint32_t c = at < A ? wl[warp][at] : 0u;
        const float xd = __shfl_sync(FULL, cd, c);
        const uint32_t xi = __shfl_sync(FULL, cid, c);
        const int xn = __shfl_sync(FULL, cn, c);
        bool hit = false;
        if (on) {
          if ((NSG || cv) && pid[p] == xi) {
            hit = true;
            if (cv) drop(c);
          } else {
            hit = occludes(xd, pd[p], pf_dist<I8>(pick_row(p), row_of(c, xi), d, I8 ? pnrm[p] : 0, xn));
            if (hit && pd[p] == xd && pid[p] != xi) amb = 1;
          }
        }
        unsigned hm = __ballot_sync(FULL, hit);
        if (G >= 2) hm |= hm >> 16;
        if (G >= 4) hm |= hm >> 8;
        am = ~hm & (A >= 32 ? FULL : (1u << A) - 1u);
        __syncwarp();
        if (lane < A && ((am >> lane) & 1u)) wl[warp][__popc(am & lt)] = c;
        A = __popc(am);
        __syncwarp();
        j += G;
      }
      if (lane == 0) wc[warp] = A;
      __syncthreads();
      // the survivors in order: each pick is tested against the rest
      while (true) {
        int fw = 0;
        while (fw < PF_NW && wc[fw] == 0) fw++;
        if (fw == PF_NW) break;  // block-uniform
        const uint32_t c = wl[fw][0], pos = ex + 32 * fw + c;
        const uint32_t xi = ki(pos);
        const float xd = kd(pos);
        __syncthreads();  // everyone has read the lists
        if (warp == fw) {
          if (lane == 0) {
            if (np > 0 && pd[np - 1] == xd && pid[np - 1] != xi) amb = 1;
            pid[np] = xi;
            pd[np] = xd;
            if (I8) pnrm[np] = (int)__ldg(a.xnorm + xi);
            gone[(pos - g0) >> 5] |= 1u << ((pos - g0) & 31);
          }
          if (f.cs) put_pick(np, cand + (size_t)f.cs * (32 * fw + c));
          const uint32_t nx = lane + 1 < A ? wl[warp][lane + 1] : 0u;
          __syncwarp();
          wl[warp][lane] = nx;
          A--;
        }
        np++;
        __syncthreads();
        if (np == a.R) {
          // a later entry of the last pick's distance could have come first
          if (tid == 0)
            for (uint32_t i = pos + 1; i < wn && kd(i) == xd; i++)
              if (ki(i) != xi) amb = 1;
          done = true;
          break;
        }
        if (A > 0) {
          const uint32_t y = lane < A ? wl[warp][lane] : 0u;
          const float yd = __shfl_sync(FULL, cd, y);
          const uint32_t yi = __shfl_sync(FULL, cid, y);
          const int yn = __shfl_sync(FULL, cn, y);
          bool hit = false;
          if (lane < A) {
            if ((NSG || cv) && xi == yi) {
              hit = true;
              if (cv) drop(y);
            } else {
              hit = occludes(yd, xd, pf_dist<I8>(pick_row(np - 1), row_of(y, yi), d, I8 ? pnrm[np - 1] : 0, yn));
              if (hit && xd == yd && xi != yi) amb = 1;
            }
          }
          const unsigned keep = __ballot_sync(FULL, lane < A && !hit);
          __syncwarp();
          if ((keep >> lane) & 1u) wl[warp][__popc(keep & lt)] = y;
          A = __popc(keep);
          __syncwarp();
        }
        if (lane == 0) wc[warp] = A;
        __syncthreads();
      }
      if (EXACT && !NSG && !done && warp == 0)  // the skipped entries, in order
        for (uint32_t w = 0; w < PF_NW; w++) {
          const uint32_t pos = ex + 32 * w + lane;
          const bool skip = pos < wend && !((gone[w] >> lane) & 1u);
          const unsigned sm = __ballot_sync(FULL, skip);
          if (skip) heap[nskip + __popc(sm & lt)] = HeapItem{kd(pos), DI{kd(pos), ki(pos)}};
          nskip += __popc(sm);
        }
      ex += 32 * PF_NW;
      __syncthreads();
    }
    if (EXACT || done) break;
    // equal distances on both sides of the bound: which were examined?
    if (tid == 0 && wbase + wend == end && wend < wn) {
      const float bd = kd(wend);
      const uint32_t bi = ki(wend);
      if (wend > 0 && kd(wend - 1) == bd) {
        for (uint32_t i = wend + 1; i < wn && kd(i) == bd; i++)
          if (ki(i) != bi) amb = 1;
        for (uint32_t i = wend; i-- > 0 && kd(i) == bd;)
          if (ki(i) != bi) amb = 1;
      }
    }
    // the least skipped keys, for the Vamana refill: the first window's
    if (!NSG && wbase == 0) {
      if (warp == 0) {
        uint32_t c = 0;
        for (uint32_t b = 0; b < wend && c < PF_SAVED; b += 32) {
          const bool skip = b + lane < wend && !((gone[b >> 5] >> lane) & 1u);
          const unsigned sm = __ballot_sync(FULL, skip);
          const uint32_t at = c + __popc(sm & lt);
          if (skip && at < PF_SAVED) saved[at] = K[b + lane];
          c += __popc(sm);
        }
        nsaved = min(c, PF_SAVED);
        all_saved = wend == end && c < PF_SAVED;
      }
    }
    wbase += wend;
    if (wbase >= end) break;
    __syncthreads();
    wn = pf_window(U, m, K, wlo, false);
    if (wn == 0) {  // a bin beyond the window's size
      if (tid == 0) amb = 1;
      break;
    }
    pf_sort<PF_WINDOW / PF_THREADS>(K);
    ex = 0;
    }
    __syncthreads();
    if (EXACT && !NSG && np < a.R && warp == 0) {
      if (lane == 0) {
        for (uint32_t k = 1; k <= nskip; k++) stl::push_heap(heap, (int)k, HeapItemLess());
        uint32_t hs = nskip;
        while (np < a.R && hs > 0) {
          bool again = false;  // clean Vamana: an id skipped twice is taken once
          for (uint32_t j = 0; cv && j < np && !again; j++) again = pid[j] == heap[0].data.i;
          if (!again) {
            pid[np] = heap[0].data.i;
            pd[np] = heap[0].data.d;
            np++;
          }
          stl::pop_heap(heap, (int)hs, HeapItemLess());
          hs--;
        }
        wc[0] = np;
      }
    } else if (!NSG && np < a.R && warp == 0) {
      // refill from the skipped min-heap (component_prune.cpp:276-279): the
      // skipped entries in ascending order
      float ld = -1.f;
      uint32_t li = 0, i = 0;
      for (; i < nsaved; i++) {
        const float xd = __uint_as_float((uint32_t)(saved[i] >> 32));
        const uint32_t xi = (uint32_t)saved[i];
        if (xd == ld && xi != li && lane == 0) amb = 1;
        if (np == a.R) {  // the entries past the last taken are looked at for a tie
          if (xd != ld) break;
          continue;
        }
        ld = xd;
        li = xi;
        bool again = false;  // clean Vamana: an id skipped twice is taken once
        if (cv)
          for (uint32_t j = lane; j < np; j += 32) again |= pid[j] == xi;
        if (__any_sync(FULL, again)) continue;
        if (lane == 0) {
          pid[np] = xi;
          pd[np] = xd;
        }
        np++;
        __syncwarp();
      }
      if (i == nsaved && !all_saved && lane == 0) amb = 1;  // more were skipped than kept here
      if (lane == 0) wc[0] = np;
    } else if (tid == 0) {
      wc[0] = np;
    }
    __syncthreads();
    if (!EXACT && amb) {
      if (tid == 0) f.redo[atomicAdd(f.nredo, 1u)] = qi;
      continue;
    }
    np = wc[0];
    for (uint32_t j = tid; j < np; j += PF_THREADS) {
      oid[j] = pid[j];
      od[j] = pd[j];
    }
    if (tid == 0) a.out_deg[node] = np;
  }
}

// ---------------------------------------------------------------- InterInsert
struct IIArgs {
  const float *base;
  const uint8_t *base8;    // byte rows (integer data, d a multiple of 16 up to 256), with their squared norms
  const float *xnorm;
  uint32_t d, n, R;
  float alpha;
  int clean;               // Vamana re-prune closest first, each candidate against its own distance
  float threshold;
  uint32_t cs;             // bytes between row vectors in shared memory (0: read where they lie)
  uint32_t spare;          // vector slots beyond the R + 1 of a re-prune
  const uint8_t *pops;     // Vamana: pops[64 N + k], the k-th item popped off a heap of N items of equal keys
  const uint32_t *p_ids;   // pruned rows (width R)
  const float *p_dist;
  const uint32_t *p_deg;
  uint32_t *s_ids;         // rows at each node's turn (width R)
  float *s_dist;
  uint32_t *s_deg;
  uint32_t *s_kept;        // (NSG) IIRow::kept of those rows
  uint32_t *f_ids;         // final rows (width R)
  float *f_dist;
  uint32_t *f_deg;
  uint32_t *done;          // level(n) + 1 once row n is at its turn, 0 before
  uint32_t *next, *maxlev; // forward: the next node, the highest level
  const unsigned long long *req;  // per target: (sender << 32 | index) sorted
  const uint32_t *req_off, *req_cnt;
  int *status;
};

constexpr int II_WARPS = 4;
constexpr uint32_t II_SPARE = 4;          // senders whose rows and vectors are loaded together
constexpr uint32_t II_POLLS = 1u << 26;   // polls of a sender's flag before the wait gives up

struct Ent3 {
  float d;
  uint32_t i;
  uint32_t slot;
};
struct Ent3Less {
  __device__ bool operator()(const Ent3 &a, const Ent3 &b) const { return a.d < b.d; }
};
struct HeapIdx {  // MinHeap item of the re-prune: key and temp index
  float key;
  uint32_t k;
};
struct HeapIdxLess {
  __host__ __device__ bool operator()(const HeapIdx &a, const HeapIdx &b) const { return a.key > b.key; }
};

// A warp holds one row: entry j in lane j % 32's set j / 32 of registers, and
// in shared memory the re-prune's scratch, the row vectors in slots, their
// norms (bytes) or ids, and the slots' pairwise distances.
struct IIWarp {
  Ent3 *tmp;      // 64
  HeapIdx *heap;  // 64 (clean Vamana)
  uint32_t *res;  // 64
  uint32_t *sid;  // NS: id of each slot's vector
  float *D;       // NS x NS
  uint8_t *V;     // NS x cs
  uint32_t NS;
};
__host__ __device__ inline uint32_t ii_slots(uint32_t R, uint32_t spare) { return R + 1 + spare; }
__host__ __device__ inline size_t ii_warp_bytes(uint32_t R, uint32_t cs, uint32_t spare) {
  const size_t S = ii_slots(R, spare);
  return 64 * sizeof(Ent3) + 64 * sizeof(HeapIdx) + 64 * 4 + ((S * 4 + 15) & ~size_t(15)) +
         ((S * S * 4 + 15) & ~size_t(15)) + S * cs;
}
__device__ inline IIWarp ii_carve(uint8_t *p, uint32_t R, uint32_t spare) {
  IIWarp w;
  w.NS = ii_slots(R, spare);
  w.tmp = reinterpret_cast<Ent3 *>(p);
  p += 64 * sizeof(Ent3);
  w.heap = reinterpret_cast<HeapIdx *>(p);
  p += 64 * sizeof(HeapIdx);
  w.res = reinterpret_cast<uint32_t *>(p);
  p += 64 * 4;
  w.sid = reinterpret_cast<uint32_t *>(p);
  p += ((size_t)w.NS * 4 + 15) & ~size_t(15);
  w.D = reinterpret_cast<float *>(p);
  p += ((size_t)w.NS * w.NS * 4 + 15) & ~size_t(15);
  w.V = p;
  return w;
}

struct IIRow {
  float d[2];
  uint32_t i[2], slot[2];
  uint32_t rs;   // entries
  bool vvalid;   // every entry has a slot holding its vector
  bool dvalid;   // D holds the slots' pairwise distances
  // (NSG) a full row, strictly ascending, no entry occluded by a nearer one:
  // what a prune or re-prune that takes R entries with distinct keys leaves.
  // Re-pruning it with s then needs only the distances to s: the nearer
  // entries are taken, s unless one of them occludes it (the row stays as it
  // was), the farther ones unless s occludes them.
  bool kept;
  Slots slots;
};

template <bool I8>
struct II {
  const IIArgs &a;
  IIWarp w;
  int lane;

  __device__ const uint8_t *vec(uint32_t slot) const {
    if (a.cs) return w.V + (size_t)slot * a.cs;
    return I8 ? a.base8 + (size_t)w.sid[slot] * a.d
              : reinterpret_cast<const uint8_t *>(a.base + (size_t)w.sid[slot] * a.d);
  }
  // starts the copy of row `id` into slot f (a warp); the caller waits.  A slot
  // given back unwaited is not taken again before a wait (wv_slots.cuh): two
  // copies into one slot could land in either order
  __device__ void stage(uint32_t f, uint32_t id) const {
    if (lane == 0) w.sid[f] = id;
    if (!a.cs) return;
    const uint8_t *src = I8 ? a.base8 + (size_t)id * a.d : reinterpret_cast<const uint8_t *>(a.base + (size_t)id * a.d);
    const uint32_t ch = (I8 ? a.d : a.d * 4) / 16;
    for (uint32_t k = lane; k < ch; k += 32) cp_async16(w.V + (size_t)f * a.cs + k * 16, src + k * 16);
  }
  __device__ void landed() const {
    cp_async_wait_all();
    __syncwarp();
  }
  __device__ uint32_t take(IIRow &r) const {
    return r.slots.take([&]() { landed(); });
  }
  __device__ float dist(uint32_t x, uint32_t y) const {
    return pf_dist<I8>(vec(x), vec(y), a.d, I8 ? (int)__ldg(a.xnorm + w.sid[x]) : 0,
                       I8 ? (int)__ldg(a.xnorm + w.sid[y]) : 0);
  }
  __device__ unsigned long long used(const IIRow &r) const {
    unsigned lo = 0, hi = 0;
#pragma unroll
    for (int h = 0; h < 2; h++)
      if (lane + 32 * h < (int)r.rs) {
        const uint32_t s = r.slot[h];
        if (s < 32) lo |= 1u << s;
        else hi |= 1u << (s - 32);
      }
    lo = __reduce_or_sync(FULL, lo);
    hi = __reduce_or_sync(FULL, hi);
    return ((unsigned long long)hi << 32) | lo;
  }
  // kept: whether the row, if full and strictly ascending, is a prune's or a
  // re-prune's result
  __device__ void load(IIRow &r, const uint32_t *ids, const float *dist, uint32_t deg, bool kept) const {
    r.rs = deg;
    r.vvalid = r.dvalid = false;
    bool asc = kept && deg == a.R;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t j = lane + 32 * h;
      r.d[h] = j < deg ? dist[j] : 0.f;
      r.i[h] = j < deg ? ids[j] : INVALID;
      r.slot[h] = 0;
    }
    float up0 = __shfl_up_sync(FULL, r.d[0], 1), up1 = __shfl_up_sync(FULL, r.d[1], 1);
    const float last0 = __shfl_sync(FULL, r.d[0], 31);
    if (lane == 0) up1 = last0;
    if (lane > 0 && lane < (int)deg) asc &= up0 < r.d[0];
    if (lane + 32 < (int)deg) asc &= up1 < r.d[1];
    r.kept = __all_sync(FULL, asc);
    r.slots.reset(w.NS);
  }
  __device__ void store(const IIRow &r, uint32_t *ids, float *dist) const {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t j = lane + 32 * h;
      if (j < r.rs) {
        ids[j] = r.i[h];
        dist[j] = r.d[h];
      }
    }
  }
  // slots and vectors for the whole row
  __device__ void give_slots(IIRow &r) const {
    r.slots.reclaim([&]() { landed(); });
#pragma unroll
    for (int h = 0; h < 2; h++) {
      unsigned long long f = r.slots.free;  // entry j takes the j-th free slot
      const uint32_t j = lane + 32 * h;
      if (j < r.rs) {
        for (uint32_t k = 0; k < j; k++) f &= f - 1;
        r.slot[h] = __ffsll(f) - 1;
      }
    }
    for (uint32_t j = 0; j < r.rs; j++) {
      const uint32_t id = j < 32 ? __shfl_sync(FULL, r.i[0], j) : __shfl_sync(FULL, r.i[1], j - 32);
      const uint32_t sl = j < 32 ? __shfl_sync(FULL, r.slot[0], j) : __shfl_sync(FULL, r.slot[1], j - 32);
      stage(sl, id);
    }
    r.slots.free &= ~used(r);
    r.vvalid = true;
  }
  __device__ void all_pairs(IIRow &r) const {
    const uint32_t np = r.rs * (r.rs - 1) / 2;
    for (uint32_t p0 = 0; p0 < np; p0 += 32) {
      const uint32_t p = p0 + lane;
      // pair p of the triangle y < x: x (x - 1) / 2 + y
      uint32_t x = (uint32_t)((1.f + sqrtf(1.f + 8.f * (float)p)) * 0.5f);
      while (x * (x - 1) / 2 > p) x--;
      while ((x + 1) * x / 2 <= p) x++;
      const uint32_t y = p - x * (x - 1) / 2;
      const uint32_t sx0 = __shfl_sync(FULL, r.slot[0], x & 31), sx1 = __shfl_sync(FULL, r.slot[1], x & 31);
      const uint32_t sy0 = __shfl_sync(FULL, r.slot[0], y & 31), sy1 = __shfl_sync(FULL, r.slot[1], y & 31);
      if (p < np) {
        const uint32_t sx = x < 32 ? sx0 : sx1, sy = y < 32 ? sy0 : sy1;
        const float dd = dist(sx, sy);
        w.D[sx * w.NS + sy] = dd;
        w.D[sy * w.NS + sx] = dd;
      }
    }
    r.dvalid = true;
    __syncwarp();
  }

  // "insert `s` (distance sd, sender index si) into this row" exactly as
  // InterInsert does to des_pool (component_refine.cpp:484-540 / 884-949 /
  // 660-720).  fs: the slot s's vector is being copied to, or INVALID
  template <int MODE>
  __device__ void apply(IIRow &r, uint32_t s, float sd, uint32_t si, uint32_t fs) const {
    constexpr bool NSG = MODE == 1;
    const uint32_t R = a.R, NS = w.NS, rs = r.rs;
    const bool h0 = lane < (int)rs, h1 = lane + 32 < (int)rs;
    auto give_back = [&]() {
      if (fs != INVALID) r.slots.give_back(fs);
    };
    if (__any_sync(FULL, (h0 && r.i[0] == s) || (h1 && r.i[1] == s))) return give_back();
    auto column = [&](uint32_t f, float (&x)[2]) {  // distances of the row's entries to slot f
      x[0] = x[1] = 0.f;
      if (h0) x[0] = dist(r.slot[0], f);
      if (h1) x[1] = dist(r.slot[1], f);
      if (r.dvalid) {
        if (h0) w.D[f * NS + r.slot[0]] = w.D[r.slot[0] * NS + f] = x[0];
        if (h1) w.D[f * NS + r.slot[1]] = w.D[r.slot[1] * NS + f] = x[1];
      }
      __syncwarp();
    };
    auto slot_for = [&]() {
      if (fs == INVALID) {
        fs = take(r);
        stage(fs, s);
      }
      landed();
    };
    if (rs + 1 <= R) {  // room: append at the sentinel
      if (r.vvalid) {
        slot_for();
        float x[2];
        if (r.dvalid) column(fs, x);
      } else {
        give_back();
        fs = 0;
      }
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (lane + 32 * h == (int)rs) {
          r.d[h] = sd;
          r.i[h] = s;
          r.slot[h] = fs;
        }
      r.rs = rs + 1;
      r.kept = false;
      return;
    }
    const unsigned n0 = __ballot_sync(FULL, h0 && r.d[0] < sd), n1 = __ballot_sync(FULL, h1 && r.d[1] < sd);
    const bool tie_s = __any_sync(FULL, (h0 && r.d[0] == sd) || (h1 && r.d[1] == sd));
    const uint32_t nnear = __popc(n0) + __popc(n1);
    const bool quick = NSG && r.kept && !tie_s;
    if (quick && nnear == rs) return give_back();  // farther than a full row's entries
    if (!r.vvalid) give_slots(r);
    slot_for();
    const unsigned long long old_slots = used(r);
    if (!quick && !r.dvalid) all_pairs(r);
    float x[2];
    column(fs, x);
    uint32_t nres = 0;
    if (quick) {
      if (__any_sync(FULL, (h0 && r.d[0] < sd && x[0] < sd) || (h1 && r.d[1] < sd && x[1] < sd))) {
        r.slots.free |= 1ull << fs;  // (its copy has landed)
        return;
      }
      // the survivors, in order, with s after the nearer ones
      const bool k0 = h0 && (r.d[0] < sd || !(x[0] < r.d[0])), k1 = h1 && (r.d[1] < sd || !(x[1] < r.d[1]));
      const unsigned m0 = __ballot_sync(FULL, k0), m1 = __ballot_sync(FULL, k1);
      const unsigned lt = (1u << lane) - 1u;
      const uint32_t p0 = __popc(m0 & lt) + (r.d[0] < sd ? 0u : 1u);
      const uint32_t p1 = __popc(m0) + __popc(m1 & lt) + (r.d[1] < sd ? 0u : 1u);
      if (k0) w.tmp[p0] = Ent3{r.d[0], r.i[0], r.slot[0]};
      if (k1) w.tmp[p1] = Ent3{r.d[1], r.i[1], r.slot[1]};
      if (lane == 0) w.tmp[nnear] = Ent3{sd, s, fs};
      __syncwarp();
      nres = min(R, (uint32_t)__popc(m0) + __popc(m1) + 1);
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (lane + 32 * h < (int)nres) {
          const Ent3 e = w.tmp[lane + 32 * h];
          r.d[h] = e.d;
          r.i[h] = e.i;
          r.slot[h] = e.slot;
        }
      r.kept = nres == R;
      // (a shorter result leaves the old entries at the remaining positions)
    } else {
      const uint32_t T = rs + 1;
      // the row and s in order: std::sort(temp_pool) (component_refine.cpp:503
      // / 901): with distinct keys the sorted array is unique, so each lane
      // places its entries by rank; tied keys take the one-lane replica
      Ent3 e0 = h0 ? Ent3{r.d[0], r.i[0], r.slot[0]} : Ent3{sd, s, fs};
      Ent3 e1 = h1 ? Ent3{r.d[1], r.i[1], r.slot[1]} : Ent3{sd, s, fs};
      uint32_t r0 = 0, r1 = 0;
      bool tie = false;
      for (uint32_t t = 0; t < T; t++) {
        const float kt = t < 32 ? __shfl_sync(FULL, e0.d, t) : __shfl_sync(FULL, e1.d, t - 32);
        r0 += kt < e0.d;
        r1 += kt < e1.d;
        tie |= (lane < T && t != lane && kt == e0.d) || (lane + 32 < T && t != lane + 32 && kt == e1.d);
      }
      const bool any_tie = __any_sync(FULL, tie);
      if (any_tie) {
        r0 = lane;
        r1 = lane + 32;
      }
      if (lane < T) w.tmp[r0] = e0;
      if (lane + 32 < T) w.tmp[r1] = e1;
      __syncwarp();
      if (any_tie && lane == 0) stl::sort(w.tmp, (int)T, Ent3Less());
      __syncwarp();
      const Ent3 p0 = lane < T ? w.tmp[lane] : Ent3{0.f, 0u, 0u};
      const Ent3 p1 = lane + 32 < T ? w.tmp[lane + 32] : Ent3{0.f, 0u, 0u};
      // bit q of o0 / o1: sorted entry q would occlude this lane's entry
      // (q before p, or any q for Vamana's farthest-first walk)
      unsigned long long o0 = 0, o1 = 0;
      const float cur = MODE == 0 && !a.clean ? w.tmp[si].d : 0.f;
      for (uint32_t q = 0; q < T; q++) {
        const Ent3 e = w.tmp[q];
        auto occ = [&](const Ent3 &p, uint32_t at) -> bool {
          if (at >= T || at == q || (MODE != 0 && q > at)) return false;
          const float dd = w.D[e.slot * NS + p.slot];
          if (MODE == 0) return __fmul_rn(a.alpha, dd) < (a.clean ? p.d : cur);
          return e.i == p.i || (MODE == 2 ? ssg_occludes(p.d, e.d, dd, a.threshold) : (dd < p.d));
        };
        if (occ(p0, lane)) o0 |= 1ull << q;
        if (T > 32 && occ(p1, lane + 32)) o1 |= 1ull << q;
      }
      auto mask_of = [&](uint32_t st) { return st < 32 ? __shfl_sync(FULL, o0, st) : __shfl_sync(FULL, o1, st - 32); };
      if (MODE == 0) {
        // compat: farthest first, every candidate against temp_pool[i].d (the
        // outer index, refine.cpp:907); clean: closest first, each candidate
        // against its own distance (the rule of PruneVAMANA)
        unsigned long long taken = 0;
        uint32_t nskip = 0;
        for (uint32_t kk = 0; kk < T && nres < R; kk++) {
          const uint32_t k = a.clean ? kk : T - 1 - kk;
          if (!(mask_of(k) & taken)) {
            taken |= 1ull << k;
            if (lane == 0) w.res[nres] = k;
            nres++;
          } else {
            if (lane == 0) w.heap[nskip] = HeapIdx{a.clean ? w.tmp[k].d : cur, k};
            nskip++;
          }
        }
        __syncwarp();
        const uint32_t take = min(R - nres, nskip);
        if (take > 0) {
          if (!a.clean) {
            // every key is `cur`: the heap's pops follow from its size
            for (uint32_t t = lane; t < take; t += 32) w.res[nres + t] = w.heap[a.pops[64 * nskip + t]].k;
          } else if (lane == 0) {
            for (uint32_t k = 1; k <= nskip; k++) stl::push_heap(w.heap, (int)k, HeapIdxLess());
            for (uint32_t t = 0; t < take; t++) {
              w.res[nres + t] = w.heap[0].k;
              stl::pop_heap(w.heap, (int)(nskip - t), HeapIdxLess());
            }
          }
          nres += take;
          __syncwarp();
        }
      } else {
        // entry 0, then each entry that no taken entry occludes, up to R
        // (component_refine.cpp:505-526)
        unsigned long long taken = 1ull;
        nres = 1;
        for (uint32_t st = 1; nres < R && st < T; st++)
          if (!(mask_of(st) & taken)) {
            taken |= 1ull << st;
            nres++;
          }
        if (lane < T && ((taken >> lane) & 1ull)) w.res[__popcll(taken & ((1ull << lane) - 1ull))] = lane;
        if (lane + 32 < T && ((taken >> (lane + 32)) & 1ull))
          w.res[__popcll(taken & ((1ull << (lane + 32)) - 1ull))] = lane + 32;
        __syncwarp();
      }
      // des_pool[t] = result[t] for t < result.size() (refine.cpp:527-530,
      // 943-946, 706-712).  Vamana results always hold R entries; an NSG
      // result may be shorter and then, with no sentinel written, the old
      // entries at positions result.size()..R-1 stay in the row; SSG writes
      // the sentinel.
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (lane + 32 * h < (int)nres) {
          const Ent3 e = w.tmp[w.res[lane + 32 * h]];
          r.d[h] = e.d;
          r.i[h] = e.i;
          r.slot[h] = e.slot;
        }
      r.kept = NSG && nres == R && !any_tie;
      if (MODE != 1) r.rs = nres;
    }
    __syncwarp();
    // the slots of entries that left (and s's, if it was not taken) are free;
    // those of pending vectors stay taken
    r.slots.free = (r.slots.free | old_slots | (1ull << fs)) & ~used(r);
  }
};

__device__ __forceinline__ uint32_t ii_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Forward: every node applies the insertions from lower ids (senders m < n
// whose row at their turn lists n), in id order, and publishes its row at its
// turn.  One cooperative launch: the warps, all resident, take nodes in id
// order and wait for a sender's flag where it is not up yet -- a sender has a
// lower id, so a running or finished warp holds it and every wait ends (each
// is bounded all the same, and a warp that gives up raises the status word
// the other waits look at).  Bound by the longest chains (a hub's re-prunes,
// one after the other).  A launch per dependency level, with a barrier after
// each level's slowest node, took 62 ms on the 200k x 128 NSG link and 79 ms
// on two 20k x 96 Vamana passes; this takes 10.4 ms and 12.7 ms (the backward
// launches 8.3 -> 4.7 and 7.5 -> 4.9 ms).
template <int MODE, bool I8>
__global__ void __launch_bounds__(II_WARPS * 32) k_ii_forward(IIArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const II<I8> t{a, ii_carve(smem + (size_t)warp * ii_warp_bytes(a.R, a.cs, a.spare), a.R, a.spare), lane};
  const uint32_t R = a.R;
  while (true) {
    uint32_t n = 0;
    if (lane == 0) n = atomicAdd(a.next, 1u);
    n = __shfl_sync(FULL, n, 0);
    if (n >= a.n) return;
    IIRow r;
    t.load(r, a.p_ids + (size_t)n * R, a.p_dist + (size_t)n * R, a.p_deg[n], MODE == 1);
    const uint32_t off = a.req_off[n], cnt = a.req_cnt[n];
    uint32_t level = 0;
    for (uint32_t r0 = 0; r0 < cnt;) {
      const uint32_t nb = min(II_SPARE, cnt - r0);
      const uint32_t m = lane < nb ? (uint32_t)(a.req[off + r0 + lane] >> 32) : 0u;
      uint32_t up = lane < nb ? ii_acquire(a.done + m) : 0u;
      // the senders that are at hand, in order; the first is waited for
      if (__shfl_sync(FULL, up, 0) == 0) {
        bool ok = true;
        if (lane == 0) {
          uint32_t polls = 0;
          while ((up = ii_acquire(a.done + m)) == 0) {
            if (++polls >= II_POLLS) {
              set_err(a.status, DEV_TIMEOUT);
              ok = false;
              break;
            }
            if ((polls & 255u) == 0 && *reinterpret_cast<volatile int *>(a.status) != 0) {
              ok = false;
              break;
            }
            __nanosleep(40);
          }
        }
        if (!__shfl_sync(FULL, ok, 0)) return;
      }
      __syncwarp();  // orders every lane's reads of the rows after the lanes' acquires (votes and shuffles do not)
      const uint32_t have = __ffs(~__ballot_sync(FULL, up != 0)) - 1;
      for (uint32_t k = 0; k < have; k++) level = max(level, __shfl_sync(FULL, up, k));
      // their rows (read past the L1, which other warps' rows may share lines with)
      uint32_t mk[II_SPARE], id[II_SPARE][2], dg[II_SPARE], fs[II_SPARE];
      float ds[II_SPARE][2];
#pragma unroll
      for (int k = 0; k < (int)II_SPARE; k++) {
        mk[k] = __shfl_sync(FULL, m, k);
        const bool on = k < (int)have;
        dg[k] = on ? __ldcg(a.s_deg + mk[k]) : 0u;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint32_t j = lane + 32 * h;
          const bool in = on && j < R;
          id[k][h] = in ? __ldcg(a.s_ids + (size_t)mk[k] * R + j) : INVALID;
          ds[k][h] = in ? __ldcg(a.s_dist + (size_t)mk[k] * R + j) : 0.f;
        }
      }
      unsigned hit[II_SPARE][2];
#pragma unroll
      for (int k = 0; k < (int)II_SPARE; k++) {
        hit[k][0] = __ballot_sync(FULL, lane < dg[k] && id[k][0] == n);
        hit[k][1] = __ballot_sync(FULL, lane + 32 < dg[k] && id[k][1] == n);
        fs[k] = INVALID;
        if (k < (int)a.spare && (hit[k][0] | hit[k][1]) && (r.vvalid || r.rs == R)) {
          fs[k] = t.take(r);
          t.stage(fs[k], mk[k]);
        }
      }
      // each position of n in a sender's row sends one insertion (an NSG row
      // can list an id twice), in position order
#pragma unroll
      for (int k = 0; k < (int)II_SPARE; k++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          unsigned hm = hit[k][h];
          while (hm) {
            const int b = __ffs(hm) - 1;
            hm &= hm - 1;
            const float sd = __shfl_sync(FULL, ds[k][h], b);
            t.template apply<MODE>(r, mk[k], sd, (uint32_t)(b + 32 * h), fs[k]);
            fs[k] = INVALID;
          }
        }
      r0 += have;
    }
    t.store(r, a.s_ids + (size_t)n * R, a.s_dist + (size_t)n * R);
    if (lane == 0) {
      a.s_deg[n] = r.rs;
      a.s_kept[n] = r.kept;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      atomicMax(a.maxlev, level);
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.done + n), "r"(level + 1) : "memory");
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");  // (a vector whose insertion was refused may still be in flight)
    __syncwarp();
  }
}

// backward: every row applies the insertions from higher ids in id order
template <int MODE, bool I8>
__global__ void __launch_bounds__(II_WARPS * 32) k_ii_backward(IIArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const II<I8> t{a, ii_carve(smem + (size_t)warp * ii_warp_bytes(a.R, a.cs, a.spare), a.R, a.spare), lane};
  const uint32_t R = a.R;
  while (true) {
    uint32_t n = 0;
    if (lane == 0) n = atomicAdd(a.next, 1u);
    n = __shfl_sync(FULL, n, 0);
    if (n >= a.n) return;
    IIRow r;
    t.load(r, a.s_ids + (size_t)n * R, a.s_dist + (size_t)n * R, a.s_deg[n], MODE == 1 && a.s_kept[n]);
    const uint32_t off = a.req_off[n], cnt = a.req_cnt[n];
    for (uint32_t r0 = 0; r0 < cnt; r0 += 32) {
      const unsigned long long key = r0 + lane < cnt ? a.req[off + r0 + lane] : 0ull;
      const uint32_t ml = (uint32_t)(key >> 32), pl = (uint32_t)key;
      const float dl = r0 + lane < cnt ? a.s_dist[(size_t)ml * R + pl] : 0.f;
      const uint32_t nb = min(32u, cnt - r0);
      uint32_t nxt = INVALID;  // the slot the next sender's vector goes to
      for (uint32_t q = 0; q < nb; q++) {
        const uint32_t m = __shfl_sync(FULL, ml, q), pos = __shfl_sync(FULL, pl, q);
        const float sd = __shfl_sync(FULL, dl, q);
        const uint32_t cur = nxt;
        nxt = INVALID;
        if (cur != INVALID) t.landed();
        if (q + 1 < nb && a.spare > 0 && r.vvalid) {
          nxt = t.take(r);
          t.stage(nxt, __shfl_sync(FULL, ml, q + 1));
        }
        t.template apply<MODE>(r, m, sd, pos, cur);
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp();
    t.store(r, a.f_ids + (size_t)n * R, a.f_dist + (size_t)n * R);
    if (lane == 0) a.f_deg[n] = r.rs;
  }
}

// requests index: count edges m -> t of rows (ids, deg) with m < t (fwd) or m > t
__global__ void k_req_count(uint32_t n, uint32_t R, const uint32_t *ids, const uint32_t *deg, int fwd, uint32_t *cnt) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  for (uint32_t j = 0; j < deg[m]; j++) {
    const uint32_t t = ids[(size_t)m * R + j];
    if (t < n && (fwd ? m < t : m > t)) atomicAdd(&cnt[t], 1u);
  }
}
__global__ void k_req_fill(uint32_t n, uint32_t R, const uint32_t *ids, const uint32_t *deg, int fwd,
                           const uint32_t *off, uint32_t *cur, unsigned long long *req) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  for (uint32_t j = 0; j < deg[m]; j++) {
    const uint32_t t = ids[(size_t)m * R + j];
    if (t < n && (fwd ? m < t : m > t))
      req[off[t] + atomicAdd(&cur[t], 1u)] = ((unsigned long long)m << 32) | j;
  }
}

// ---------------------------------------------------------------- Propagation2
// ComponentCandidatePropagation2::CandidateInner (component_candidate.cpp:90-109):
// the pool takes the unseen neighbours of the node's neighbours, walking the
// node's row and each neighbour's row in order, and stops at L entries.  One
// warp per node handles a neighbour row 32 entries at a time: a lane's entry
// is new when the seen-set lacks it and no lower lane holds the same id; the
// first (L - size) new entries, in lane order, are appended and marked.  The
// seen-set is an open-addressing hash in shared memory (at most L + 1 of its
// 2^k >= 2(L + 1) words are ever used, so a probe always ends).
constexpr int P2_WARPS_MAX = 8;
constexpr uint32_t P2_EMPTY = 0xffffffffu;

struct Prop2Args {
  const float *base;
  uint32_t d, n;
  const uint32_t *g_ids, *g_deg;
  uint32_t gw;
  uint32_t n0, cnt;   // nodes [n0, n0 + cnt)
  uint32_t L;
  uint32_t hwords;    // seen-set words per warp (power of two)
  DI *vis;            // cnt x vcap pools
  uint32_t vcap;
  uint32_t *vcnt;
  int *status;
};

__device__ __forceinline__ uint32_t p2_slot(uint32_t v, uint32_t mask) { return (v * 0x9E3779B1u) & mask; }

__device__ __forceinline__ bool p2_find(const uint32_t *H, uint32_t mask, uint32_t v) {
  uint32_t h = p2_slot(v, mask);
  for (uint32_t t = 0; t <= mask; t++, h = (h + 1) & mask) {
    const uint32_t x = H[h];
    if (x == v) return true;
    if (x == P2_EMPTY) return false;
  }
  return false;
}

__device__ __forceinline__ void p2_insert(uint32_t *H, uint32_t mask, uint32_t v) {
  uint32_t h = p2_slot(v, mask);
  for (uint32_t t = 0; t <= mask; t++, h = (h + 1) & mask) {
    const uint32_t old = atomicCAS(H + h, P2_EMPTY, v);
    if (old == P2_EMPTY || old == v) return;
  }
}

__global__ void k_prop2(Prop2Args a) {
  extern __shared__ uint32_t p2_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  uint32_t *H = p2_smem + (size_t)warp * a.hwords;
  const uint32_t mask = a.hwords - 1;
  const unsigned lt = (1u << lane) - 1u;
  for (uint32_t qi = blockIdx.x * wpb + warp; qi < a.cnt; qi += gridDim.x * wpb) {
    const uint32_t q = a.n0 + qi;
    DI *pool = a.vis + (size_t)qi * a.vcap;
    for (uint32_t k = lane; k < a.hwords; k += 32) H[k] = P2_EMPTY;
    __syncwarp();
    if (lane == 0) p2_insert(H, mask, q);
    __syncwarp();
    uint32_t size = 0;
    const uint32_t qdeg = min(a.g_deg[q], a.gw);
    for (uint32_t i = 0; i < qdeg && size < a.L; i++) {
      const uint32_t nid = a.g_ids[(size_t)q * a.gw + i];
      if (nid >= a.n) {
        if (lane == 0) set_err(a.status, DEV_BAD_ID);
        continue;
      }
      const uint32_t ndeg = min(a.g_deg[nid], a.gw);
      for (uint32_t b = 0; b < ndeg && size < a.L; b += 32) {
        const uint32_t j = b + lane;
        uint32_t v = j < ndeg ? a.g_ids[(size_t)nid * a.gw + j] : P2_EMPTY;
        if (j < ndeg && v >= a.n) {
          set_err(a.status, DEV_BAD_ID);
          v = P2_EMPTY;
        }
        bool fresh = v != P2_EMPTY && !p2_find(H, mask, v);
        const unsigned same = __match_any_sync(FULL, v);
        fresh = fresh && (same & lt) == 0;  // the lowest lane holding v speaks for it
        const unsigned newm = __ballot_sync(FULL, fresh);
        const uint32_t take = min((uint32_t)__popc(newm), a.L - size);
        const uint32_t rank = __popc(newm & lt);
        __syncwarp();  // every lookup of this batch precedes its insertions
        if (fresh && rank < take) {
          pool[size + rank] = DI{0.f, v};
          p2_insert(H, mask, v);
        }
        size += take;
        __syncwarp();
      }
    }
    // distances in the reference's order, one lane per entry
    for (uint32_t j = lane; j < size; j += 32) pool[j].d = l2g(a.base, a.d, q, pool[j].i);
    if (lane == 0) a.vcnt[qi] = size;
    __syncwarp();
  }
}

// ---------------------------------------------------------------- SSG conn
// smallest reached node whose row has a free slot (deg < R); *out starts at ~0
__global__ void k_first_open(const uint32_t *bits, const uint32_t *deg, uint32_t n, uint32_t R, uint32_t *out) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (((bits[j >> 5] >> (j & 31)) & 1u) && deg[j] < R) {
      atomicMin(out, j);
      return;  // later j of this thread are larger
    }
  }
}

// one repair of ConnSSGDFS (component_conn.cpp:205-221): node u = the smallest
// unreached id; the first reached node j with a free slot gets the edge
// j -> u (distance in the reference's order); u is marked and becomes the
// frontier.  u >= n ends the root's pass (frontier size 0).
__global__ void k_ssg_repair(const float *base, uint32_t d, uint32_t n, uint32_t w, uint32_t R, uint32_t *ids,
                             float *dist, uint32_t *deg, const uint32_t *u_in, uint32_t *j_in, uint32_t *bits,
                             uint32_t *front, uint32_t *nfront, uint32_t *added) {
  if (threadIdx.x != 0) return;
  const uint32_t u = *u_in, j = *j_in;
  *j_in = 0xffffffffu;
  if (u >= n) {
    *nfront = 0;
    return;
  }
  if (j < n && deg[j] < R) {
    const uint32_t pos = deg[j];
    ids[(size_t)j * w + pos] = u;
    dist[(size_t)j * w + pos] = l2g(base, d, j, u);
    deg[j] = pos + 1;
    *added += 1;
  }
  bits[u >> 5] |= 1u << (u & 31);
  front[0] = u;
  *nfront = 1;
}

// the first row whose degree is above w or that holds an id >= n (a warp a row)
__global__ void k_conn_check(const uint32_t *ids, const uint32_t *deg, uint32_t n, uint32_t w, uint32_t *bad) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
    const uint32_t dg = deg[v];
    bool b = dg > w;
    for (uint32_t j = lane; j < min(dg, w); j += 32) b |= ids[(size_t)v * w + j] >= n;
    if (__any_sync(FULL, b) && lane == 0) atomicMin(bad, v);
  }
}

// rows list[0..m) (a warp a row)
__global__ void k_conn_gather(const uint32_t *ids, uint32_t w, const uint32_t *list, uint32_t m, uint32_t *out) {
  const int lane = threadIdx.x & 31;
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= m) return;
  const uint32_t *src = ids + (size_t)list[r] * w;
  for (uint32_t j = lane; j < w; j += 32) out[(size_t)r * w + j] = src[j];
}

__global__ void k_mark_root(uint32_t *bits, uint32_t r, uint32_t *front) {
  bits[r >> 5] |= 1u << (r & 31);
  front[0] = r;
}

}  // namespace

// ================================================================ host side
namespace {

int run_build_search(wv_ctx *c, const float *d_queries, uint32_t nq, const uint32_t *d_seeds, uint32_t seed_stride,
                     uint32_t L, const uint32_t *gids, const uint32_t *gdeg, uint32_t gw, DI *vis, uint32_t *vcnt,
                     uint32_t vcap, uint32_t *out_ids, uint32_t K, bool distinct, uint32_t vlimit = 0) {
  if (vlimit == 0) vlimit = vcap;
  const uint32_t cap = gw + 32;
  int blocks = search_grid(c->d, L, cap, c->device);
  WV_CHECK(c, blocks > 0, WV_ERR_LIMIT, "candidate search cannot run with d=%u L=%u width=%u", c->d, L, gw);
  size_t slots = (size_t)blocks * search_warps_per_block();
  size_t words = (c->n + 31) / 32;
  if (slots > c->vis_slots || words != c->vis_words) {
    c->visited.release();
    c->touched.release();
    WV_CUDA(c, c->visited.ensure(slots * words * 4));
    WV_CUDA(c, c->touched.ensure(slots * words * 4));
    WV_CUDA(c, cudaMemsetAsync(c->visited.p, 0, slots * words * 4, c->stream));
    c->vis_slots = slots;
    c->vis_words = words;
  }
  WV_CUDA(c, cudaMemsetAsync(c->misc.p, 0, 32, c->stream));
  SearchArgs a{};
  a.base = c->base.as<float>();
  a.n = c->n;
  a.d = c->d;
  a.gids = gids;
  a.gdeg = gdeg;
  a.gw = gw;
  a.distinct = distinct;
  a.queries = d_queries;
  a.nq = nq;
  a.seeds = d_seeds;
  a.seed_stride = seed_stride;
  a.L = L;
  a.K = K;
  a.Lmax = L;
  a.out_ids = out_ids;
  a.out_stride = K;
  a.visited = c->visited.as<uint32_t>();
  a.touched = c->touched.as<uint32_t>();
  a.words = (uint32_t)words;
  a.cap = cap;
  a.next_query = c->d_next();
  a.status = c->d_status();
  a.vis = vis;
  a.vcnt = vcnt;
  a.vcap = vcap;
  a.vlimit = vlimit;
  a.int_exact = c->base_int;
  a.xnorm = c->xnorm.as<float>();
  a.base8 = c->base_int && c->d <= SEARCH_I8_D ? c->base8.as<uint8_t>() : nullptr;
  int nb = (int)std::min<size_t>((size_t)blocks, ((size_t)nq + search_warps_per_block() - 1) / search_warps_per_block());
  WV_CUDA(c, launch_search_exact(a, std::max(nb, 1), c->stream));
  return WV_OK;
}

// seen-set words per warp for pool size L, and the warps per block that fit
uint32_t prop2_hwords(uint32_t L) {
  uint32_t h = 64;
  while (h < 2 * (L + 1)) h <<= 1;
  return h;
}

int run_prop2(wv_ctx *c, uint32_t n0, uint32_t cnt, uint32_t L, DI *vis, uint32_t *vcnt, uint32_t vcap) {
  Prop2Args a{};
  a.base = c->base.as<float>();
  a.d = c->d;
  a.n = c->n;
  a.g_ids = c->fg_ids.as<uint32_t>();
  a.g_deg = c->fg_deg.as<uint32_t>();
  a.gw = c->fg_w;
  a.n0 = n0;
  a.cnt = cnt;
  a.L = L;
  a.hwords = prop2_hwords(L);
  a.vis = vis;
  a.vcap = vcap;
  a.vcnt = vcnt;
  a.status = c->d_status();
  const size_t per_warp = (size_t)a.hwords * 4;
  const int wpb = (int)std::max<size_t>(1, std::min<size_t>(P2_WARPS_MAX, (96u << 10) / per_warp));
  const size_t smem = per_warp * wpb;
  WV_CUDA(c, cudaFuncSetAttribute(k_prop2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int blocks = (int)std::min<size_t>(((size_t)cnt + wpb - 1) / wpb, (size_t)c->sms * 16);
  k_prop2<<<std::max(blocks, 1), wpb * 32, smem, c->stream>>>(a);
  WV_CUDA(c, cudaGetLastError());
  return WV_OK;
}

// float threshold = std::cos(A / 180 * kPi) (component_prune.cpp:92-93,
// component_refine.cpp:640-641): float quotient, double product and cosine
float ssg_threshold(float A) {
  const double kPi = std::acos(-1.0);
  return (float)std::cos((double)(A / 180) * kPi);
}

}  // namespace

int link_gpu(wv_ctx *c, const LinkParams &p, LinkStats *st) {
  const bool ssg = p.mode == LinkMode::SSG, vamana = p.mode == LinkMode::VAMANA;
  WV_CHECK(c, c->n > 0 && c->fg_n == c->n, WV_ERR_STATE, "the link needs the base and a candidate graph");
  WV_CHECK(c, p.R >= 1 && p.R <= LINK_MAX_R, WV_ERR_LIMIT, "R_refine=%u: this build supports 1..%u", p.R, LINK_MAX_R);
  if (ssg)
    WV_CHECK(c, p.L >= 1 && p.L <= (1u << 13), WV_ERR_ARG, "L_refine=%u out of range", p.L);
  else
    WV_CHECK(c, p.L >= 1 && p.L < c->n && p.L <= SEARCH_MAX_L, WV_ERR_ARG, "L_refine=%u out of range", p.L);
  WV_CHECK(c, c->fg_w <= SEARCH_MAX_WIDTH, WV_ERR_LIMIT, "candidate graph width %u above %u", c->fg_w,
           SEARCH_MAX_WIDTH);
  WV_CHECK(c, c->d % 4 == 0, WV_ERR_LIMIT, "dimension %u is not a multiple of 4", c->d);
  LinkStats local;
  LinkStats &S = st ? *st : local;
  S = LinkStats();
  cudaError_t e = cudaSuccess;
  const uint32_t n = c->n, R = p.R, gw = c->fg_w;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, c->stream);
  // host copies of what the host-side draws need
  std::vector<uint32_t> hdeg(n);
  int repeats = 1;
  WV_CUDA(c, rows_repeat(c->fg_ids.as<uint32_t>(), c->fg_deg.as<uint32_t>(), n, gw, c->d_repeats(), &repeats, c->sms,
                         c->stream));
  WV_CUDA(c, cudaMemcpyAsync(hdeg.data(), c->fg_deg.p, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  auto host_row = [&](uint32_t v, std::vector<uint32_t> &out) -> int {
    out.resize(hdeg[v]);
    if (hdeg[v])
      WV_CUDA(c, cudaMemcpy(out.data(), c->fg_ids.as<uint32_t>() + (size_t)v * gw, hdeg[v] * 4, cudaMemcpyDeviceToHost));
    return WV_OK;
  };
  float *center = c->buf<float>("center", c->d, &e);
  uint32_t *seed1 = c->buf<uint32_t>("seed1", p.L, &e);
  uint32_t *one = c->buf<uint32_t>("one", 4, &e);
  WV_CUDA(c, e);
  // ---- entry point (ComponentRefineEntryCentroid::EntryInner); SSG has none
  // (its RefineInner leaves the entry step out) and draws no rand() here
  uint32_t ep = 0;
  if (!ssg) {
  // EntryCentroid's FP32 column sums in the reference's order (i ascending)
  WV_CUDA(c, col_chain(c->base.as<float>(), n, c->d, true, center, c->stream));
  ep = (uint32_t)c->rnd.next() % n;
  if (p.entry_L == 0) {
    ep = 0;  // get_neighbors with L = 0 leaves retset[0] value-initialised
  } else {
    std::vector<uint32_t> row, sd(p.entry_L);
    int rc = host_row(ep, row);
    if (rc) return rc;
    draw_seeds_row(c->rnd, p.entry_L, n, row.data(), (uint32_t)row.size(), sd.data());
    WV_CUDA(c, cudaMemcpyAsync(seed1, sd.data(), p.entry_L * 4, cudaMemcpyHostToDevice, c->stream));
    DI *v1 = c->buf<DI>("vis1", (size_t)n + p.entry_L + 64, &e);
    WV_CUDA(c, e);
    rc = run_build_search(c, center, 1, seed1, p.entry_L, p.entry_L, c->fg_ids.as<uint32_t>(),
                          c->fg_deg.as<uint32_t>(), gw, v1, one + 1, n + p.entry_L + 64, one, 1, !repeats);
    if (rc) return rc;
    WV_CUDA(c, cudaMemcpyAsync(&ep, one, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  }
  S.ep = ep;
  // ---- candidates + prune, in chunks of nodes
  uint32_t *p_ids = c->buf<uint32_t>("lk_pids", (size_t)n * R, &e);
  float *p_dist = c->buf<float>("lk_pdist", (size_t)n * R, &e);
  uint32_t *p_deg = c->buf<uint32_t>("lk_pdeg", n, &e);
  WV_CUDA(c, e);
  std::vector<uint32_t> ep_row;
  if (!ssg) {
    int rc = host_row(ep, ep_row);
    if (rc) return rc;
  }
  const bool shared_seeds = ssg || p.L <= ep_row.size();  // no rand() fill needed
  // SSG pools hold at most L candidates plus the node's row
  uint32_t vcap = ssg ? p.L + gw : std::max<uint32_t>(2048, 8 * p.L) + gw;
  const uint32_t CH = std::min<uint32_t>(n, 1u << 17);
  std::vector<uint32_t> hseeds;
  uint32_t *dseeds = c->buf<uint32_t>("lk_seeds", (size_t)(shared_seeds ? 1 : CH) * p.L, &e);
  WV_CUDA(c, e);
  if (shared_seeds && !ssg)
    WV_CUDA(c, cudaMemcpyAsync(dseeds, ep_row.data(), p.L * 4, cudaMemcpyHostToDevice, c->stream));
  const int prune_blocks = c->sms * 4;  // of the EXACT launch
  const float threshold = ssg ? ssg_threshold(p.A) : 0.f;
  for (uint32_t n0 = 0; n0 < n; n0 += CH) {
    const uint32_t cnt = std::min(CH, n - n0);
    if (!shared_seeds) {
      hseeds.resize((size_t)cnt * p.L);
      for (uint32_t q = 0; q < cnt; q++) {
        // the fill draws rand() % N until L ids are taken (candidate.cpp:25-31)
        draw_seeds_row(c->rnd, p.L, n, ep_row.data(), (uint32_t)ep_row.size(), hseeds.data() + (size_t)q * p.L);
      }
      WV_CUDA(c, cudaMemcpyAsync(dseeds, hseeds.data(), (size_t)cnt * p.L * 4, cudaMemcpyHostToDevice, c->stream));
    }
    while (true) {
      DI *vis = c->buf<DI>("lk_vis", (size_t)cnt * vcap, &e);
      uint32_t *vcnt = c->buf<uint32_t>("lk_vcnt", cnt, &e);
      int *gscr = c->buf<int>("lk_gscr", prune_blocks * (2 * (size_t)vcap + 256), &e);
      HeapItem *hscr = c->buf<HeapItem>("lk_hscr", prune_blocks * (size_t)vcap, &e);
      WV_CUDA(c, e);
      int rc = ssg ? run_prop2(c, n0, cnt, p.L, vis, vcnt, vcap)
                   : run_build_search(c, c->base.as<float>() + (size_t)n0 * c->d, cnt, dseeds,
                                      shared_seeds ? 0 : p.L, p.L, c->fg_ids.as<uint32_t>(),
                                      c->fg_deg.as<uint32_t>(), gw, vis, vcnt, vcap, nullptr, 1, !repeats,
                                      vcap - ((vamana && !p.clean) ? 0 : gw));
      if (rc) return rc;
      int st0 = 0;
      WV_CUDA(c, cudaMemcpyAsync(&st0, c->d_status(), 4, cudaMemcpyDeviceToHost, c->stream));
      WV_CUDA(c, cudaStreamSynchronize(c->stream));
      if (st0 == DEV_OVERFLOW && !ssg) {  // a visit list outgrew vcap: redo the chunk with room
        WV_CUDA(c, cudaMemsetAsync(c->d_status(), 0, 4, c->stream));
        vcap = vcap * 2;
        continue;
      }
      rc = check_device_status(c, "candidate search");
      if (rc) return rc;
      PruneArgs pa{};
      pa.base = c->base.as<float>();
      pa.d = c->d;
      pa.n = n;
      pa.vis = vis;
      pa.vcnt = vcnt;
      pa.vcap = vcap;
      pa.n0 = n0;
      pa.cnt = cnt;
      pa.R = R;
      pa.alpha = p.alpha;
      pa.clean = p.clean ? 1 : 0;
      pa.maxc = p.C;
      pa.threshold = threshold;
      pa.g_ids = c->fg_ids.as<uint32_t>();
      pa.g_deg = c->fg_deg.as<uint32_t>();
      pa.gw = gw;
      pa.gscr = gscr;
      pa.hscr = hscr;
      pa.out_ids = p_ids;
      pa.out_dist = p_dist;
      pa.out_deg = p_deg;
      pa.status = c->d_status();
      // integer data with byte rows (d a multiple of 16 up to 256): the pair
      // distances as exact integers (WV_LINK_PRUNE=fp32 keeps the
      // exact-order FP32 sums)
      const char *pr_env = getenv("WV_LINK_PRUNE");
      const bool i8 = c->base_int && c->base8.p && !(pr_env && std::string(pr_env) == "fp32");
      pa.xnorm = i8 ? c->xnorm.as<float>() : nullptr;
      uint32_t *lists = c->buf<uint32_t>("lk_plist", PF_SIZES * (size_t)cnt, &e);
      uint32_t *lcnts = c->buf<uint32_t>("lk_plcnt", PF_SIZES, &e);
      WV_CUDA(c, e);
      WV_CUDA(c, cudaMemsetAsync(lcnts, 0, PF_SIZES * 4, c->stream));
      PruneFast pf{};
      pf.base8 = i8 ? c->base8.as<uint8_t>() : nullptr;
      // rows in shared memory where 4 warps' candidates and the picks fit
      // (an odd multiple of 16 bytes apart: no bank conflicts)
      const uint32_t rb16 = i8 ? c->d : c->d * 4;
      auto row_stride = [&](bool exact) -> uint32_t {
        const uint32_t cs = rb16 / 16 % 2 ? rb16 : rb16 + 16;
        return pf_smem(pf.keys, cs, R, exact) <= 200 * 1024 ? cs : 0;
      };
      pf.redo = lists + (PF_SIZES - 1) * (size_t)cnt;
      pf.nredo = lcnts + PF_SIZES - 1;
      auto launch = [&](auto exact) -> cudaError_t {
        constexpr bool X = decltype(exact)::value;
        const size_t sm = pf_smem(pf.keys, pf.cs, R, X);
        auto go = [&](auto kern) -> cudaError_t {
          cudaError_t x = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
          int per = 0;
          if (x == cudaSuccess) x = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, PF_THREADS, sm);
          if (x != cudaSuccess) return x;
          const uint32_t grid = X ? (uint32_t)prune_blocks : (uint32_t)(c->sms * std::max(per, 1) * 4);
          kern<<<std::min<uint32_t>(cnt, grid), PF_THREADS, sm, c->stream>>>(pa, pf);
          return cudaGetLastError();
        };
        if (ssg) return i8 ? go(k_prune_block<2, true, X>) : go(k_prune_block<2, false, X>);
        if (!vamana) return i8 ? go(k_prune_block<1, true, X>) : go(k_prune_block<1, false, X>);
        return i8 ? go(k_prune_block<0, true, X>) : go(k_prune_block<0, false, X>);
      };
      for (int l = 0; l < PF_SIZES; l++) {
        pf.keys = pf_keys(l);
        pf.cs = row_stride(false);
        pf.list = l ? lists + (size_t)(l - 1) * cnt : nullptr;
        pf.nlist = l ? lcnts + (l - 1) : nullptr;
        pf.more = l < PF_SIZES - 1 ? lists + (size_t)l * cnt : nullptr;
        pf.nmore = l < PF_SIZES - 1 ? lcnts + l : nullptr;
        WV_CUDA(c, launch(std::false_type{}));
      }
      pf.keys = pf_keys(1);
      pf.cs = row_stride(true);
      pf.list = pf.redo;
      pf.nlist = pf.nredo;
      WV_CUDA(c, launch(std::true_type{}));
      WV_CUDA(c, cudaGetLastError());
      rc = check_device_status(c, "prune");
      if (rc) return rc;
      break;
    }
  }
  // ---- InterInsert
  uint32_t *done = c->buf<uint32_t>("lk_done", n, &e);
  uint32_t *kept = c->buf<uint32_t>("lk_kept", n, &e);
  uint32_t *iis = c->buf<uint32_t>("lk_iis", 4, &e);  // [0] next node, [1] highest level
  uint32_t *rcnt = c->buf<uint32_t>("lk_rcnt", n, &e);
  uint32_t *roff = c->buf<uint32_t>("lk_roff", n + 1, &e);
  uint32_t *rcur = c->buf<uint32_t>("lk_rcur", n, &e);
  uint32_t *scan_tmp = c->buf<uint32_t>("lk_scan", scan_scratch_words((size_t)n + 1), &e);
  unsigned long long *req = c->buf<unsigned long long>("lk_req", (size_t)n * R + 1, &e);
  uint32_t *s_ids = c->buf<uint32_t>("lk_sids", (size_t)n * R, &e);
  float *s_dist = c->buf<float>("lk_sdist", (size_t)n * R, &e);
  uint32_t *s_deg = c->buf<uint32_t>("lk_sdeg", n, &e);
  uint8_t *pops = c->buf<uint8_t>("lk_pops", 65 * 64, &e);
  WV_CUDA(c, e);
  const int nb = (int)((n + 255) / 256);
  // forward request lists from the pruned rows, sorted by sender
  WV_CUDA(c, cudaMemsetAsync(rcnt, 0, (size_t)n * 4, c->stream));
  WV_CUDA(c, cudaMemsetAsync(rcur, 0, (size_t)n * 4, c->stream));
  k_req_count<<<nb, 256, 0, c->stream>>>(n, R, p_ids, p_deg, 1, rcnt);
  WV_CUDA(c, exclusive_scan_u32(rcnt, roff, n, scan_tmp, c->stream));
  k_req_fill<<<nb, 256, 0, c->stream>>>(n, R, p_ids, p_deg, 1, roff, rcur, req);
  int rc = segsort_u64(c, req, roff, rcnt, n);
  if (rc) return rc;
  std::vector<uint8_t> hpops;
  if (vamana && !p.clean) {
    // the order in which libstdc++'s heap steps pop N items of equal keys
    hpops.assign(65 * 64, 0);
    for (int N = 1; N <= 64; N++) {
      HeapIdx h[64];
      for (int k = 0; k < N; k++) {
        h[k] = HeapIdx{0.f, (uint32_t)k};
        stl::push_heap(h, k + 1, HeapIdxLess());
      }
      for (int k = 0; k < N; k++) {
        hpops[64 * N + k] = (uint8_t)h[0].k;
        stl::pop_heap(h, N - k, HeapIdxLess());
      }
    }
    WV_CUDA(c, cudaMemcpyAsync(pops, hpops.data(), hpops.size(), cudaMemcpyHostToDevice, c->stream));
  }
  const bool ii8 = c->base_int && c->base8.p;
  IIArgs ia{};
  ia.base = c->base.as<float>();
  ia.base8 = ii8 ? c->base8.as<uint8_t>() : nullptr;
  ia.xnorm = ii8 ? c->xnorm.as<float>() : nullptr;
  ia.d = c->d;
  ia.n = n;
  ia.R = R;
  ia.alpha = p.alpha;
  ia.clean = p.clean ? 1 : 0;
  ia.threshold = threshold;
  ia.spare = std::min(II_SPARE, LINK_MAX_R - R);
  // row vectors in shared memory when they fit (an odd multiple of 16 bytes
  // apart: no bank conflicts), else read where they lie
  const uint32_t irb = ii8 ? c->d : c->d * 4;
  ia.cs = irb / 16 % 2 ? irb : irb + 16;
  if (II_WARPS * ii_warp_bytes(R, ia.cs, ia.spare) > 200 * 1024) ia.cs = 0;
  ia.pops = pops;
  ia.p_ids = p_ids;
  ia.p_dist = p_dist;
  ia.p_deg = p_deg;
  ia.s_ids = s_ids;
  ia.s_dist = s_dist;
  ia.s_deg = s_deg;
  ia.s_kept = kept;
  ia.done = done;
  ia.next = iis;
  ia.maxlev = iis + 1;
  ia.req = req;
  ia.req_off = roff;
  ia.req_cnt = rcnt;
  ia.status = c->d_status();
  const size_t ii_smem = II_WARPS * ii_warp_bytes(R, ia.cs, ia.spare);
  auto ii_launch = [&](auto kern, bool coop) -> cudaError_t {
    cudaError_t x = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ii_smem);
    int per = 0;
    if (x == cudaSuccess) x = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, II_WARPS * 32, ii_smem);
    if (x != cudaSuccess) return x;
    const dim3 grid(std::max(1u, std::min<uint32_t>((uint32_t)(per * c->sms), (n + II_WARPS - 1) / II_WARPS)));
    void *args[] = {&ia};
    if (coop) return cudaLaunchCooperativeKernel((const void *)kern, grid, dim3(II_WARPS * 32), args, ii_smem, c->stream);
    return cudaLaunchKernel((const void *)kern, grid, dim3(II_WARPS * 32), args, ii_smem, c->stream);
  };
  WV_CUDA(c, cudaMemsetAsync(done, 0, (size_t)n * 4, c->stream));
  WV_CUDA(c, cudaMemsetAsync(iis, 0, 16, c->stream));
  if (ssg) WV_CUDA(c, ii8 ? ii_launch(k_ii_forward<2, true>, true) : ii_launch(k_ii_forward<2, false>, true));
  else if (vamana) WV_CUDA(c, ii8 ? ii_launch(k_ii_forward<0, true>, true) : ii_launch(k_ii_forward<0, false>, true));
  else WV_CUDA(c, ii8 ? ii_launch(k_ii_forward<1, true>, true) : ii_launch(k_ii_forward<1, false>, true));
  rc = check_device_status(c, "inter-insert");
  if (rc) return rc;
  uint32_t maxlev = 0;
  WV_CUDA(c, cudaMemcpyAsync(&maxlev, iis + 1, 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  S.levels = maxlev + 1;
  // backward request lists from the snapshots, sorted by sender
  WV_CUDA(c, cudaMemsetAsync(rcnt, 0, (size_t)n * 4, c->stream));
  WV_CUDA(c, cudaMemsetAsync(rcur, 0, (size_t)n * 4, c->stream));
  k_req_count<<<nb, 256, 0, c->stream>>>(n, R, s_ids, s_deg, 0, rcnt);
  WV_CUDA(c, exclusive_scan_u32(rcnt, roff, n, scan_tmp, c->stream));
  k_req_fill<<<nb, 256, 0, c->stream>>>(n, R, s_ids, s_deg, 0, roff, rcur, req);
  rc = segsort_u64(c, req, roff, rcnt, n);
  if (rc) return rc;
  // final rows (width R) replace the build graph
  WV_CUDA(c, c->fg_ids.ensure((size_t)n * R * 4));
  WV_CUDA(c, c->fg_dist.ensure((size_t)n * R * 4));
  WV_CUDA(c, c->fg_deg.ensure((size_t)n * 4));
  ia.f_ids = c->fg_ids.as<uint32_t>();
  ia.f_dist = c->fg_dist.as<float>();
  ia.f_deg = c->fg_deg.as<uint32_t>();
  WV_CUDA(c, cudaMemsetAsync(iis, 0, 16, c->stream));
  if (ssg) WV_CUDA(c, ii8 ? ii_launch(k_ii_backward<2, true>, false) : ii_launch(k_ii_backward<2, false>, false));
  else if (vamana) WV_CUDA(c, ii8 ? ii_launch(k_ii_backward<0, true>, false) : ii_launch(k_ii_backward<0, false>, false));
  else WV_CUDA(c, ii8 ? ii_launch(k_ii_backward<1, true>, false) : ii_launch(k_ii_backward<1, false>, false));
  rc = check_device_status(c, "inter-insert");
  if (rc) return rc;
  c->fg_w = R;
  c->fg_ep = ep;
  c->fg_has_ep = !ssg;
  c->fg_eps.clear();
  cudaEventRecord(e1, c->stream);
  cudaEventSynchronize(e1);
  cudaEventElapsedTime(&S.ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return WV_OK;
}

// The conn edges root -> id at row position pos, applied on the device: the
// id, the distance compare(base[root], base[id]) (ComponentConnNSGDFS::
// findroot, component_conn.cpp:94-97) and the row's degree.
struct ConnEdge {
  uint32_t root, id, pos;
};

__global__ void k_conn_edges(const float *base, uint32_t d, const ConnEdge *e, uint32_t ne, uint32_t *gids,
                             float *gdist, uint32_t *gdeg, uint32_t w) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += gridDim.x * blockDim.x) {
    const ConnEdge x = e[i];
    gids[(size_t)x.root * w + x.pos] = x.id;
    gdist[(size_t)x.root * w + x.pos] = l2g(base, d, x.root, x.id);
    atomicMax(gdeg + x.root, x.pos + 1);
  }
}

// rows ids[0..B) of the base, packed (the queries of a batch of searches)
__global__ void k_conn_rows(const float *base, uint32_t d, const uint32_t *ids, uint32_t B, float *out) {
  const size_t total = (size_t)B * d;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x)
    out[t] = base[(size_t)ids[t / d] * d + t % d];
}

// the rows (width w0) re-laid out with width w1, entries past a row's
// degree zero
__global__ void k_conn_relayout(const uint32_t *ids, const float *dist, const uint32_t *deg, uint32_t n, uint32_t w0,
                                uint32_t w1, uint32_t *ids1, float *dist1) {
  const size_t total = (size_t)n * w1;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)(t / w1), j = (uint32_t)(t % w1);
    const bool in = j < w0 && j < deg[v];
    ids1[t] = in ? ids[(size_t)v * w0 + j] : 0u;
    dist1[t] = in ? dist[(size_t)v * w0 + j] : 0.f;
  }
}

int conn_dfs_gpu(wv_ctx *c, uint32_t L_refine, uint32_t *added) {
  // ComponentConnNSGDFS::tree_grow (component_conn.cpp:14-98).
  //
  // Which nodes get linked, and in which order, follows from the rows alone:
  // everything reachable from a flagged node is flagged, so the DFS after a
  // repair leaves the new root only through the new edge, the flagged set
  // after repair k is the closure of ep and the first k linked nodes over
  // the rows as they were, and the next linked node is the smallest
  // unflagged id.  The host walks that first: ft[x] is the repair after
  // which x is flagged (0: the walk from ep), tgt the linked nodes in order.
  //
  // The roots come from greedy searches (get_neighbors from ep's row) that
  // read the rows with the edges added so far and draw rand() for their
  // seeds.  They run as one batch over the linked nodes still to do, all on
  // the rows and the rand() stream as they stand at the batch's start (the
  // seeds from a copy of the stream).  The host then takes the results in
  // repair order and accepts search k while (a) the real stream, at k's
  // turn, gives the same seeds (the fallback's extra draws and an edge
  // appended to a short ep row change them) and (b) none of the rows it
  // read -- its seeds' and its visits' -- got an edge earlier in the batch.
  // The first search that fails starts the next batch, so every accepted
  // search is the one the serial walk runs and the first of a batch is
  // always accepted.  With a caller's rand() function (the stream cannot be
  // copied) each batch is one search.
  //
  // The rows stay on the device (edges appended there, widths changed by a
  // copy kernel).  What ep reaches does not depend on the walk's order, so it
  // is found there, level by level; the host walks the other nodes, few as a
  // rule, on a copy of their rows, and keeps ep's row with its new edges, for
  // the seeds.  With all rows copied to the host, checked and walked there the
  // 200k x 128 NSG link (104 ms) took 15 ms more.
  const uint32_t n = c->n, ep = c->fg_ep, w0 = c->fg_w;
  uint32_t w = w0;
  constexpr uint32_t NONE = 0xffffffffu;
  *added = 0;
  cudaError_t e0 = cudaSuccess;
  const uint32_t words = (n + 31) / 32;
  uint32_t *bits = c->buf<uint32_t>("cn_bits", words, &e0);
  uint32_t *fa = c->buf<uint32_t>("cn_fa", n, &e0);
  uint32_t *fb = c->buf<uint32_t>("cn_fb", n, &e0);
  uint32_t *cnt = c->buf<uint32_t>("cn_cnt", 4, &e0);  // [0] frontier size, [1] first bad row
  WV_CUDA(c, e0);
  std::vector<uint32_t> deg(n);
  uint32_t bad = NONE;
  WV_CUDA(c, cudaMemsetAsync(cnt, 0xff, 8, c->stream));
  k_conn_check<<<c->sms * 8, 256, 0, c->stream>>>(c->fg_ids.as<uint32_t>(), c->fg_deg.as<uint32_t>(), n, w0, cnt + 1);
  WV_CUDA(c, cudaGetLastError());
  WV_CUDA(c, cudaMemcpyAsync(&bad, cnt + 1, 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaMemcpyAsync(deg.data(), c->fg_deg.p, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  if (bad != NONE) {
    WV_CHECK(c, deg[bad] <= w0, WV_ERR_STATE, "row %u: degree %u > width %u", bad, deg[bad], w0);
    WV_CHECK(c, false, WV_ERR_STATE, "row %u holds an id >= n", bad);
  }
  std::vector<uint32_t> hbits(words), rest;
  WV_CUDA(c, cudaMemsetAsync(bits, 0, (size_t)words * 4, c->stream));
  k_mark_root<<<1, 1, 0, c->stream>>>(bits, ep, fa);
  for (uint32_t nf = 1; nf;) {
    WV_CUDA(c, cudaMemsetAsync(cnt, 0, 4, c->stream));
    const uint32_t blocks = std::min<uint32_t>((nf + 7) / 8, (uint32_t)c->sms * 32);
    k_bfs_level<<<blocks, 256, 0, c->stream>>>(c->fg_ids.as<uint32_t>(), c->fg_deg.as<uint32_t>(), w0, n, fa, nf, bits,
                                               fb, cnt, c->d_status());
    WV_CUDA(c, cudaGetLastError());
    WV_CUDA(c, cudaMemcpyAsync(&nf, cnt, 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    std::swap(fa, fb);
  }
  WV_CUDA(c, cudaMemcpyAsync(hbits.data(), bits, (size_t)words * 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  for (uint32_t v = 0; v < n; v++)
    if (!(hbits[v >> 5] >> (v & 31) & 1u)) rest.push_back(v);
  if (rest.empty()) return WV_OK;
  // the rows of the nodes ep does not reach
  const uint32_t nr = (uint32_t)rest.size();
  uint32_t *drows = c->buf<uint32_t>("cn_rows", (size_t)nr * w0, &e0);
  WV_CUDA(c, e0);
  std::vector<uint32_t> ids((size_t)nr * w0), at(n, NONE), ep_row(deg[ep]);
  WV_CUDA(c, cudaMemcpyAsync(fa, rest.data(), (size_t)nr * 4, cudaMemcpyHostToDevice, c->stream));
  k_conn_gather<<<(nr + 7) / 8, 256, 0, c->stream>>>(c->fg_ids.as<uint32_t>(), w0, fa, nr, drows);
  WV_CUDA(c, cudaGetLastError());
  WV_CUDA(c, cudaMemcpyAsync(ids.data(), drows, ids.size() * 4, cudaMemcpyDeviceToHost, c->stream));
  if (deg[ep])
    WV_CUDA(c, cudaMemcpyAsync(ep_row.data(), c->fg_ids.as<uint32_t>() + (size_t)ep * w0, (size_t)deg[ep] * 4,
                               cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  // the walk: flag times and the linked nodes
  std::vector<uint32_t> ft(n, 0), tgt, st;
  for (uint32_t i = 0; i < nr; i++) {
    at[rest[i]] = i;
    ft[rest[i]] = NONE;
  }
  auto walk = [&](uint32_t start, uint32_t t) {  // DFS (component_conn.cpp:31-57)
    st.assign(1, start);
    ft[start] = t;
    uint32_t tmp = start;
    while (!st.empty()) {
      uint32_t next = NONE;
      for (uint32_t j = 0; j < deg[tmp]; j++)
        if (ft[ids[(size_t)at[tmp] * w0 + j]] == NONE) {
          next = ids[(size_t)at[tmp] * w0 + j];
          break;
        }
      if (next == NONE) {
        st.pop_back();
        if (st.empty()) break;
        tmp = st.back();
        continue;
      }
      tmp = next;
      ft[tmp] = t;
      st.push_back(tmp);
    }
  };
  for (uint32_t v : rest) {  // findroot's first unflagged id only grows
    if (ft[v] != NONE) continue;
    tgt.push_back(v);
    walk(v, (uint32_t)tgt.size());
  }
  const uint32_t m = (uint32_t)tgt.size();
  // re-lays the device rows out with width nw
  auto relayout = [&](uint32_t nw) -> int {
    DevBuf &ti = c->work["conn_ri"], &td = c->work["conn_rd"];
    WV_CUDA(c, ti.ensure((size_t)n * nw * 4));
    WV_CUDA(c, td.ensure((size_t)n * nw * 4));
    const size_t total = (size_t)n * nw;
    const int nb = (int)std::min<size_t>((total + 255) / 256, (size_t)c->sms * 16);
    k_conn_relayout<<<nb, 256, 0, c->stream>>>(c->fg_ids.as<uint32_t>(), c->fg_dist.as<float>(),
                                                c->fg_deg.as<uint32_t>(), n, w, nw, ti.as<uint32_t>(),
                                                td.as<float>());
    WV_CUDA(c, cudaGetLastError());
    std::swap(c->fg_ids, ti);
    std::swap(c->fg_dist, td);
    w = nw;
    c->fg_w = w;
    return WV_OK;
  };
  // accepted edges not yet in the device rows
  std::vector<ConnEdge> edges;
  auto flush = [&]() -> int {
    if (edges.empty()) return WV_OK;
    const uint32_t ne = (uint32_t)edges.size();
    cudaError_t e2 = cudaSuccess;
    ConnEdge *de = c->buf<ConnEdge>("conn_e", ne, &e2);
    WV_CUDA(c, e2);
    WV_CUDA(c, cudaMemcpyAsync(de, edges.data(), (size_t)ne * sizeof(ConnEdge), cudaMemcpyHostToDevice, c->stream));
    k_conn_edges<<<(ne + 127) / 128, 128, 0, c->stream>>>(c->base.as<float>(), c->d, de, ne, c->fg_ids.as<uint32_t>(),
                                                          c->fg_dist.as<float>(), c->fg_deg.as<uint32_t>(), w);
    WV_CUDA(c, cudaGetLastError());
    edges.clear();
    return WV_OK;
  };
  int rc = relayout(w + 16);  // spare width for the edges this pass adds
  if (rc) return rc;
  const bool own = c->rnd.fn == nullptr;
  // searches per batch at most (WV_CONN_BATCH=1 runs them one at a time)
  uint32_t batch_max = 4096;
  if (const char *be = getenv("WV_CONN_BATCH")) batch_max = (uint32_t)std::min(4096L, std::max(1L, atol(be)));
  uint32_t vcap = L_refine + std::max<uint32_t>(1024, 16 * L_refine);
  std::vector<uint32_t> sd, real(L_refine), vcnt_h;
  std::vector<DI> vis_h, hv;
  std::vector<char> changed(n, 0);
  std::vector<uint32_t> changed_list;
  uint32_t k0 = 0;
  while (k0 < m) {
    rc = flush();  // the rows as they stand
    if (rc) return rc;
    for (uint32_t v : changed_list) changed[v] = 0;
    changed_list.clear();
    const uint32_t B = own ? std::min(m - k0, batch_max) : 1;
    sd.resize((size_t)B * L_refine);
    if (own) {
      RandSource spec = c->rnd;
      for (uint32_t b = 0; b < B; b++)
        draw_seeds_row(spec, L_refine, n, ep_row.data(), (uint32_t)ep_row.size(), sd.data() + (size_t)b * L_refine);
    } else {
      draw_seeds_row(c->rnd, L_refine, n, ep_row.data(), (uint32_t)ep_row.size(), sd.data());
    }
    cudaError_t e = cudaSuccess;
    uint32_t *dseed = c->buf<uint32_t>("conn_seed", (size_t)B * L_refine, &e);
    uint32_t *dtg = c->buf<uint32_t>("conn_tg", B, &e);
    float *dq = c->buf<float>("conn_q", (size_t)B * c->d, &e);
    uint32_t *dvc = c->buf<uint32_t>("conn_vc", B, &e);
    uint32_t *dout = c->buf<uint32_t>("conn_out", B, &e);
    WV_CUDA(c, e);
    WV_CUDA(c, cudaMemcpyAsync(dseed, sd.data(), (size_t)B * L_refine * 4, cudaMemcpyHostToDevice, c->stream));
    WV_CUDA(c, cudaMemcpyAsync(dtg, tgt.data() + k0, (size_t)B * 4, cudaMemcpyHostToDevice, c->stream));
    {
      const size_t total = (size_t)B * c->d;
      const int nb = (int)std::min<size_t>((total + 255) / 256, (size_t)c->sms * 8);
      k_conn_rows<<<nb, 256, 0, c->stream>>>(c->base.as<float>(), c->d, dtg, B, dq);
      WV_CUDA(c, cudaGetLastError());
    }
    DI *vis = nullptr;
    while (true) {  // get_neighbors(base[id]) from ep's row (component_conn.cpp:100-160)
      vis = c->buf<DI>("conn_vis", (size_t)B * vcap, &e);
      WV_CUDA(c, e);
      rc = run_build_search(c, dq, B, dseed, L_refine, L_refine, c->fg_ids.as<uint32_t>(), c->fg_deg.as<uint32_t>(),
                            w, vis, dvc, vcap, dout, 1, false);
      if (rc) return rc;
      int st0 = 0;
      WV_CUDA(c, cudaMemcpyAsync(&st0, c->d_status(), 4, cudaMemcpyDeviceToHost, c->stream));
      WV_CUDA(c, cudaStreamSynchronize(c->stream));
      if (st0 == DEV_OVERFLOW) {  // a visit list outgrew vcap: redo the batch with room
        WV_CUDA(c, cudaMemsetAsync(c->d_status(), 0, 4, c->stream));
        vcap *= 2;
        continue;
      }
      rc = check_device_status(c, "conn search");
      if (rc) return rc;
      break;
    }
    vcnt_h.resize(B);
    vis_h.resize((size_t)B * vcap);
    WV_CUDA(c, cudaMemcpyAsync(vcnt_h.data(), dvc, (size_t)B * 4, cudaMemcpyDeviceToHost, c->stream));
    WV_CUDA(c, cudaStreamSynchronize(c->stream));
    // the visit lists come back in growing chunks, each list only as far as
    // the chunk's longest: a batch is usually cut after a few searches
    uint32_t have = 0, chunk = 16;
    uint32_t acc = 0;
    for (uint32_t b = 0; b < B; b++) {
      if (b == have) {
        const uint32_t hi = std::min(B, have + chunk);
        uint32_t wmax = 1;
        for (uint32_t q = have; q < hi; q++) wmax = std::max(wmax, std::min(vcnt_h[q], vcap));
        WV_CUDA(c, cudaMemcpy2DAsync(vis_h.data() + (size_t)have * vcap, (size_t)vcap * sizeof(DI),
                                     vis + (size_t)have * vcap, (size_t)vcap * sizeof(DI), (size_t)wmax * sizeof(DI),
                                     hi - have, cudaMemcpyDeviceToHost, c->stream));
        WV_CUDA(c, cudaStreamSynchronize(c->stream));
        have = hi;
        chunk *= 2;
      }
      const uint32_t k = k0 + b, u = tgt[k];
      const uint32_t nv = std::min(vcnt_h[b], vcap);
      const DI *v = vis_h.data() + (size_t)b * vcap;
      bool stale = false;
      for (uint32_t j = 0; j < nv && !stale; j++) stale = v[j].i < n && changed[v[j].i];
      if (stale) break;
      if (own) {
        const RandSource keep = c->rnd;
        draw_seeds_row(c->rnd, L_refine, n, ep_row.data(), (uint32_t)ep_row.size(), real.data());
        if (!std::equal(real.begin(), real.end(), sd.data() + (size_t)b * L_refine)) {
          c->rnd = keep;
          break;
        }
      }
      // the pool: the expansion visits (the seeds are not part of it), sorted
      hv.assign(v + std::min(nv, L_refine), v + nv);
      stl::sort(hv.data(), (int)hv.size(), DILess());
      uint32_t root = NONE;
      for (auto &x : hv)
        if (x.i < n && ft[x.i] <= k) {
          root = x.i;
          break;
        }
      if (root == NONE) {
        while (true) {
          const uint32_t rid = (uint32_t)c->rnd.next() % n;
          if (ft[rid] <= k) {
            root = rid;
            break;
          }
        }
      }
      if (deg[root] == w) {
        rc = flush();
        if (rc) return rc;
        rc = relayout(w + 16);
        if (rc) return rc;
      }
      const uint32_t pos = deg[root]++;
      edges.push_back(ConnEdge{root, u, pos});
      if (root == ep) ep_row.push_back(u);
      if (!changed[root]) {
        changed[root] = 1;
        changed_list.push_back(root);
      }
      (*added)++;
      acc++;
    }
    WV_CHECK(c, acc > 0, WV_ERR_STATE, "conn: the first search of a batch was not accepted");
    k0 += acc;
  }
  rc = flush();
  if (rc) return rc;
  uint32_t nw = 1;  // trim to the widest row
  for (uint32_t v = 0; v < n; v++) nw = std::max(nw, deg[v]);
  if (nw != w) rc = relayout(nw);
  if (rc) return rc;
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  return WV_OK;
}

int conn_ssg_gpu(wv_ctx *c, uint32_t n_try, uint32_t R, std::vector<uint32_t> &eps, uint32_t *added) {
  // ComponentConnSSGDFS::ConnInner (component_conn.cpp:169-225).  The roots
  // are the first n_try ids of std::random_shuffle(0..n-1) on rand()
  // (libstdc++: for i = 1..n-1 swap ids[i] with ids[rand() % (i + 1)]).
  // From each root a breadth-first walk; while nodes stay unreached, the
  // smallest unreached id u is linked from the first reached node with a free
  // slot (if any), marked, and walked from.  Reach does not depend on the
  // walk's order, so the walk runs level-synchronously on the GPU.
  const uint32_t n = c->n, w = c->fg_w;
  WV_CHECK(c, n_try >= 1 && n_try <= n, WV_ERR_ARG, "n_try=%u out of range (n=%u)", n_try, n);
  WV_CHECK(c, R <= w, WV_ERR_ARG, "range %u above the row width %u", R, w);
  std::vector<uint32_t> perm(n);
  for (uint32_t i = 0; i < n; i++) perm[i] = i;
  for (uint32_t i = 1; i < n; i++) {
    const uint32_t j = (uint32_t)c->rnd.next() % (i + 1);
    if (i != j) std::swap(perm[i], perm[j]);
  }
  eps.assign(perm.begin(), perm.begin() + n_try);
  cudaError_t e = cudaSuccess;
  const uint32_t words = (n + 31) / 32;
  uint32_t *bits = c->buf<uint32_t>("sc_bits", words, &e);
  uint32_t *fa = c->buf<uint32_t>("sc_fa", n, &e);
  uint32_t *fb = c->buf<uint32_t>("sc_fb", n, &e);
  uint32_t *cnt = c->buf<uint32_t>("sc_cnt", 8, &e);  // [0] frontier size, [1] u, [2] j, [3] added
  WV_CUDA(c, e);
  WV_CUDA(c, cudaMemsetAsync(cnt, 0, 32, c->stream));
  WV_CUDA(c, cudaMemsetAsync(cnt + 2, 0xff, 4, c->stream));
  uint32_t *ids = c->fg_ids.as<uint32_t>(), *deg = c->fg_deg.as<uint32_t>();
  float *dist = c->fg_dist.as<float>();
  const int scan_blocks = c->sms * 4;
  for (uint32_t t = 0; t < n_try; t++) {
    WV_CUDA(c, cudaMemsetAsync(bits, 0, (size_t)words * 4, c->stream));
    k_mark_root<<<1, 1, 0, c->stream>>>(bits, eps[t], fa);
    uint32_t nf = 1;
    for (;;) {
      while (nf) {
        WV_CUDA(c, cudaMemsetAsync(cnt, 0, 4, c->stream));
        const uint32_t blocks = std::min<uint32_t>((nf + 7) / 8, (uint32_t)c->sms * 32);
        k_bfs_level<<<blocks, 256, 0, c->stream>>>(ids, deg, w, n, fa, nf, bits, fb, cnt, c->d_status());
        WV_CUDA(c, cudaGetLastError());
        WV_CUDA(c, cudaMemcpyAsync(&nf, cnt, 4, cudaMemcpyDeviceToHost, c->stream));
        WV_CUDA(c, cudaStreamSynchronize(c->stream));
        std::swap(fa, fb);
      }
      k_first_unreached<<<1, 1024, 0, c->stream>>>(bits, n, cnt + 1);
      k_first_open<<<scan_blocks, 256, 0, c->stream>>>(bits, deg, n, R, cnt + 2);
      k_ssg_repair<<<1, 32, 0, c->stream>>>(c->base.as<float>(), c->d, n, w, R, ids, dist, deg, cnt + 1,
                                            cnt + 2, bits, fa, cnt, cnt + 3);
      WV_CUDA(c, cudaGetLastError());
      WV_CUDA(c, cudaMemcpyAsync(&nf, cnt, 4, cudaMemcpyDeviceToHost, c->stream));
      WV_CUDA(c, cudaStreamSynchronize(c->stream));
      if (!nf) break;
    }
  }
  WV_CUDA(c, cudaMemcpyAsync(added, cnt + 3, 4, cudaMemcpyDeviceToHost, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));
  return check_device_status(c, "ssg conn");
}

}  // namespace wv

// SEARCH_ENTRY_RAND seeds on the device.
//
// ComponentSearchEntryRand::SearchEntryInner (src/component_search_entry.cpp
// :9-30) seeds a std::mt19937 with one rand() per query and draws the query's
// L entry ids with GenRandom (include/weavess/util.h:13-27):
//   addr[i] = rng() % (N - L) for i < L; sort; addr[i] = max(addr[i],
//   addr[i-1] + 1); off = rng() % N; addr[i] = (addr[i] + off) % N.
// The host draws the rand() values in query order (the reference's shared
// stream) and ships 4 bytes per query; one warp per query then seeds its
// mt19937 (lane 0 runs the seeding recurrence), twists it as often as L + 1
// outputs need, sorts the L residues (bitonic, ints: any correct sort gives
// the same array), bumps duplicates with a prefix maximum of
// addr[i] - i, and writes the ids.  Identical to the host draw
// (wv_host.cpp gen_random) bit for bit.
#include <cstdint>
#include <algorithm>
#include <vector>

#include "wv_common.cuh"
#include "wv_ctx.h"
#include "wv_mt.cuh"
#include "wv_seeds.h"

namespace wv {
namespace {

constexpr int SEED_WARPS = 4;

__global__ void __launch_bounds__(SEED_WARPS * 32)
    k_seeds_rand(const uint32_t *sv, uint32_t nq, const uint32_t *nq_dev, const uint32_t *Lq, uint32_t L0,
                 uint32_t Lmax, uint32_t N, uint32_t *out, uint32_t stride, int *status) {
  const uint32_t Pmax = pow2_ge(Lmax);
  extern __shared__ uint32_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t *mt = sm + (size_t)warp * (624 + Pmax + 1);
  uint32_t *key = mt + 624;
  const uint32_t q = blockIdx.x * SEED_WARPS + warp;
  if (q >= (nq_dev ? min(*nq_dev, nq) : nq)) return;  // warp-uniform
  const uint32_t L = Lq ? Lq[q] : L0;
  if (L > Lmax || L >= N) {  // the host checks; a device-side beam list may not
    if (lane == 0) set_err(status, DEV_OVERFLOW);
    return;
  }
  if (lane == 0) {
    uint32_t x = sv[q];
    mt[0] = x;
    for (uint32_t i = 1; i < 624; i++) {
      x = mt_seed_next(x, i);
      mt[i] = x;
    }
  }
  __syncwarp();
  // outputs 0..L-1 are the residues, output L the offset
  const uint32_t span = N - L;
  for (uint32_t base = 0; base <= L; base += 624) {
    mt_twist_warp(mt, lane);
    for (uint32_t i = lane; i < 624 && base + i <= L; i += 32) {
      const uint32_t v = mt_temper(mt[i]);
      key[base + i] = base + i < L ? v % span : v % N;
    }
    __syncwarp();
  }
  const uint32_t off = key[L];
  __syncwarp();
  warp_gen_random_tail(key, L, off, N, out + (size_t)q * stride, lane);
}

// The same for beams up to 32 PR, QB queries per block of 8 warps.  The
// seeding recurrence (624 dependent steps) runs for the block's queries at
// once, a query per lane of the first warp; then a warp per query at a time
// twists only as far as L + 1 outputs reach, sorts the residues in registers
// (entry i in lane i % 32's register i / 32) and takes the prefix maximum.
// Bound by that serial chain (5 us) and instruction issue: 10,000 queries at
// L = 256 take 44 us, a warp per query with the recurrence on one lane and the
// sort in shared memory took 111 us.
constexpr int SB_WARPS = 8, SB_QUERIES = 32;

template <int PR>
__global__ void __launch_bounds__(SB_WARPS * 32)
    k_seeds_block(const uint32_t *sv, uint32_t nq_max, const uint32_t *nq_dev, const uint32_t *Lq, uint32_t L0,
                  uint32_t Lmax, uint32_t N, uint32_t *out, uint32_t stride, uint32_t QB, int *status) {
  extern __shared__ uint32_t sm[];  // 624 rows of QB state words, rows an odd number of words apart
  const uint32_t st = QB | 1u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t nq = nq_dev ? min(*nq_dev, nq_max) : nq_max, q0 = blockIdx.x * QB;
  if (q0 >= nq) return;  // block-uniform
  const uint32_t qn = min(QB, nq - q0);
  if (warp == 0 && lane < (int)qn) {
    uint32_t x = sv[q0 + lane];
    sm[lane] = x;
#pragma unroll 8
    for (uint32_t i = 1; i < 624; i++) {
      x = mt_seed_next(x, i);
      sm[i * st + lane] = x;
    }
  }
  __syncthreads();
  for (uint32_t qi = warp; qi < qn; qi += SB_WARPS) {
    const uint32_t q = q0 + qi, L = Lq ? Lq[q] : L0;
    if (L > Lmax || L >= N) {  // the host checks; a device-side beam list may not
      if (lane == 0) set_err(status, DEV_OVERFLOW);
      continue;
    }
    uint32_t *mt = sm + qi;
    // the twist of the words outputs 0..L come from (L < 624): [0, 227) read
    // old words only, [227, 454) the new words i - 227, [454, 623) those of
    // the second part, word 623 the new word 0
    const uint32_t need = L + 1;
    for (uint32_t lo = 0; lo < need; lo += 227) {
      const uint32_t hi = min(min(lo + 227, need), 623u);
      uint32_t v[8];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const uint32_t i = lo + lane + 32 * r;
        if (i < hi) v[r] = mt_mix(mt[i * st], mt[(i + 1) * st], lo ? mt[(i - 227) * st] : mt[(i + 397) * st]);
      }
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const uint32_t i = lo + lane + 32 * r;
        if (i < hi) mt[i * st] = v[r];
      }
      __syncwarp();
    }
    const uint32_t span = N - L;
    uint32_t key[PR];
#pragma unroll
    for (int r = 0; r < PR; r++) {
      const uint32_t i = lane + 32 * r;
      key[r] = i < L ? mt_temper(mt[i * st]) % span : 0xffffffffu;
    }
    const uint32_t off = mt_temper(mt[L * st]) % N;
    // ascending bitonic sort of 32 PR keys
#pragma unroll
    for (int k = 2; k <= 32 * PR; k <<= 1)
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        if (j >= 32) {
#pragma unroll
          for (int r = 0; r < PR; r++)
            if ((r & (j >> 5)) == 0) {
              const int o = r | (j >> 5);
              const bool up = ((32 * r) & k) == 0;
              const uint32_t a = min(key[r], key[o]), b = max(key[r], key[o]);
              key[r] = up ? a : b;
              key[o] = up ? b : a;
            }
        } else {
#pragma unroll
          for (int r = 0; r < PR; r++) {
            const uint32_t o = __shfl_xor_sync(FULL, key[r], j);
            const bool up = ((lane + 32 * r) & k) == 0;
            key[r] = ((lane & j) == 0) == up ? min(key[r], o) : max(key[r], o);
          }
        }
      }
    // a_i = i + max_{j <= i}(v_j - j); v_j + L - j is positive and below N
    uint32_t carry = 0;
#pragma unroll
    for (int r = 0; r < PR; r++) {
      const uint32_t i = lane + 32 * r;
      uint32_t u = i < L ? key[r] + (L - i) : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, u, o);
        if (lane >= o) u = max(u, y);
      }
      u = max(u, carry);
      carry = __shfl_sync(FULL, u, 31);
      if (i < L) {
        const uint32_t a = u - (L - i);
        out[(size_t)q * stride + i] = a >= N - off ? a - (N - off) : a + off;
      }
    }
    __syncwarp();
  }
}

__global__ void k_put_roots(uint32_t nq, const uint32_t *d_nq, const uint32_t *roots, uint32_t nr, uint32_t *out,
                            uint32_t stride) {
  const uint32_t n = d_nq ? min(nq, *d_nq) : nq;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < (size_t)n * nr; t += (size_t)gridDim.x * blockDim.x)
    out[(t / nr) * stride + t % nr] = roots[t % nr];
}

}  // namespace

int put_roots_device(wv_ctx *c, uint32_t nq, const uint32_t *d_nq, uint32_t *d_out, uint32_t stride) {
  const uint32_t nr = (uint32_t)c->eps.size();
  WV_CHECK(c, nr > 0, WV_ERR_STATE, "the search graph has no SSG roots");
  WV_CHECK(c, nr <= stride, WV_ERR_ARG, "%u roots do not fit a seed row of %u", nr, stride);
  if (nq == 0) return WV_OK;
  cudaError_t e = cudaSuccess;
  uint32_t *d_roots = c->buf<uint32_t>("sd_roots", nr, &e);
  WV_CUDA(c, e);
  WV_CUDA(c, cudaMemcpyAsync(d_roots, c->eps.data(), (size_t)nr * 4, cudaMemcpyHostToDevice, c->stream));
  const size_t total = (size_t)nq * nr;
  const int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)c->sms * 8);
  k_put_roots<<<blocks, 256, 0, c->stream>>>(nq, d_nq, d_roots, nr, d_out, stride);
  WV_CUDA(c, cudaGetLastError());
  WV_CUDA(c, cudaStreamSynchronize(c->stream));  // the roots' host copy may change after this call
  return WV_OK;
}

size_t seeds_rand_smem(uint32_t Lmax) { return (size_t)SEED_WARPS * (624 + pow2_ge(Lmax) + 1) * 4; }

cudaError_t seeds_rand_launch(const uint32_t *d_sv, uint32_t nq, const uint32_t *d_nq, const uint32_t *d_L,
                              uint32_t L, uint32_t Lmax, uint32_t N, uint32_t *d_out, uint32_t stride, int *d_status,
                              int sms, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  if (Lmax <= 512) {
    // two blocks per SM first, then up to a warp of queries each
    const uint32_t fill = 2 * (uint32_t)sms, QB = std::min<uint32_t>(SB_QUERIES, (nq + fill - 1) / fill);
    const size_t smem = (size_t)624 * (QB | 1u) * 4;
    auto go = [&](auto k) -> cudaError_t {
      const cudaError_t x = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (x != cudaSuccess) return x;
      k<<<(nq + QB - 1) / QB, SB_WARPS * 32, smem, s>>>(d_sv, nq, d_nq, d_L, L, Lmax, N, d_out, stride, QB, d_status);
      return cudaGetLastError();
    };
    return Lmax <= 128 ? go(k_seeds_block<4>) : Lmax <= 256 ? go(k_seeds_block<8>) : go(k_seeds_block<16>);
  }
  const size_t smem = seeds_rand_smem(Lmax);
  cudaError_t e = cudaFuncSetAttribute(k_seeds_rand, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const uint32_t blocks = (nq + SEED_WARPS - 1) / SEED_WARPS;
  k_seeds_rand<<<blocks, SEED_WARPS * 32, smem, s>>>(d_sv, nq, d_nq, d_L, L, Lmax, N, d_out, stride, d_status);
  return cudaGetLastError();
}

// the per-query rand() values, drawn in query order, and the device draw
int draw_seeds_rand_device(wv_ctx *c, uint32_t nq, const uint32_t *d_L, uint32_t L, uint32_t Lmax, uint32_t *d_out,
                           uint32_t stride) {
  WV_CHECK(c, Lmax < c->n, WV_ERR_ARG, "L=%u must be smaller than n=%u", Lmax, c->n);
  WV_CHECK(c, Lmax <= SEED_MAX_L, WV_ERR_LIMIT, "L=%u above %u", Lmax, SEED_MAX_L);
  std::vector<uint32_t> sv(nq);
  for (uint32_t q = 0; q < nq; q++) sv[q] = (uint32_t)c->rnd.next();
  cudaError_t e = cudaSuccess;
  uint32_t *d_sv = c->buf<uint32_t>("sd_sv", nq, &e);
  WV_CUDA(c, e);
  WV_CUDA(c, cudaMemcpyAsync(d_sv, sv.data(), (size_t)nq * 4, cudaMemcpyHostToDevice, c->stream));
  WV_CUDA(c, cudaStreamSynchronize(c->stream));  // sv is consumed before it goes out of scope
  WV_CUDA(c, seeds_rand_launch(d_sv, nq, nullptr, d_L, L, Lmax, c->n, d_out, stride, c->d_status(), c->sms, c->stream));
  return WV_OK;
}

}  // namespace wv

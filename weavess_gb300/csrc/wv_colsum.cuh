// Column sums of a row-major n x N FP32 matrix with the rows added in
// ascending order, one chain of FP32 adds per column: the value a sequential
// loop gives, where the order of the additions shows in the result (the
// centroid of component_entry.cpp:9-40, the bias gradients).
#pragma once
#include <cstdint>

#include "wv_common.cuh"

namespace wv {

// A block takes 32 columns.  Warp 0 adds the rows of one shared-memory tile
// while eight warps fetch the next, so the chain of adds does not wait for each
// load; a tile's load latency bounds the kernel: 200k x 128 in 1.4 ms, against
// 8 ms with a thread per column loading inside its chain.
constexpr int CC_ROWS = 256, CC_LOADERS = 8, CC_THREADS = 32 * (CC_LOADERS + 1);
constexpr size_t CC_SMEM = 2 * (size_t)CC_ROWS * 32 * sizeof(float);

// mean: the sums are divided by n
static __global__ void __launch_bounds__(CC_THREADS) k_col_chain(const float *__restrict__ x, size_t n, uint32_t N,
                                                                 int mean, float *out) {
  extern __shared__ float cc_sm[];  // 2 x CC_ROWS x 32
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t col = blockIdx.x * 32 + lane;
  auto fill = [&](int buf, size_t r0) {
    float v[CC_ROWS / CC_LOADERS];
    const int w = warp - 1;
#pragma unroll
    for (int i = 0; i < CC_ROWS / CC_LOADERS; i++) {
      const size_t r = r0 + (size_t)i * CC_LOADERS + w;
      v[i] = col < N && r < n ? __ldg(x + r * N + col) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < CC_ROWS / CC_LOADERS; i++)
      cc_sm[((size_t)buf * CC_ROWS + i * CC_LOADERS + w) * 32 + lane] = v[i];
  };
  if (warp > 0) fill(0, 0);
  __syncthreads();
  float s = 0.f;
  int buf = 0;
  for (size_t r0 = 0; r0 < n; r0 += CC_ROWS, buf ^= 1) {
    if (warp == 0) {
      const float *t = cc_sm + (size_t)buf * CC_ROWS * 32 + lane;
      if (n - r0 >= CC_ROWS) {
#pragma unroll 32
        for (int r = 0; r < CC_ROWS; r++) s = __fadd_rn(s, t[r * 32]);
      } else {
        for (size_t r = 0; r < n - r0; r++) s = __fadd_rn(s, t[r * 32]);
      }
    } else if (r0 + CC_ROWS < n) {
      fill(buf ^ 1, r0 + CC_ROWS);
    }
    __syncthreads();
  }
  if (warp == 0 && col < N) out[col] = mean ? __fdiv_rn(s, (float)n) : s;
}

inline cudaError_t col_chain(const float *x, size_t n, uint32_t N, bool mean, float *out, cudaStream_t st) {
  if (N == 0) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(k_col_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CC_SMEM);
  if (e != cudaSuccess) return e;
  k_col_chain<<<(N + 31) / 32, CC_THREADS, CC_SMEM, st>>>(x, n, N, mean ? 1 : 0, out);
  return cudaGetLastError();
}

}  // namespace wv

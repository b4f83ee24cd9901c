// The throughput form's kernel variants (wv_beam.cuh), compiled in a
// translation unit each: together they took two minutes of compiler time.
#pragma once
#include <cuda_runtime.h>

#include "wv_search.h"

namespace wv {

// COOP: several warps per query; DISTINCT: no row of the graph repeats an id
template <bool COOP, bool DISTINCT>
struct BeamKernels {
  static int blocks_per_sm(int threads, size_t smem);  // of the variant's kernels, the least
  static void launch(int blocks, int threads, size_t smem, cudaStream_t stream, const SearchArgs &b);
};

}  // namespace wv

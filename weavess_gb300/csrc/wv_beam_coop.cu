// The throughput form's variant (wv_beam.cuh): several warps per query.
#include "wv_beam.cuh"

namespace wv {

template struct BeamKernels<true, false>;

}  // namespace wv

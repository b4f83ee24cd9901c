// The throughput form's variant (wv_beam.cuh): several warps per query, rows that list no id twice.
#include "wv_beam.cuh"

namespace wv {

template struct BeamKernels<true, true>;

}  // namespace wv

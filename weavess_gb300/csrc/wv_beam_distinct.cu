// The throughput form's variant (wv_beam.cuh): rows that list no id twice.
#include "wv_beam.cuh"

namespace wv {

template struct BeamKernels<false, true>;

}  // namespace wv

// Launch of the throughput form (wv_beam.cuh), and its plain variant.
#include "wv_beam.cuh"

namespace wv {

template struct BeamKernels<false, false>;
extern template struct BeamKernels<false, true>;
extern template struct BeamKernels<true, false>;
extern template struct BeamKernels<true, true>;

uint32_t beam_cap(uint32_t gw, uint32_t parents) {
  const uint32_t e = std::min(std::max(parents, 1u), BEAM_MAX_PARENTS);
  return e * gw + 32;
}

bool beam_shape_ok(const SearchShape &sh) {
  // several warps per query: one query group per block
  return (sh.wpb == 1 || sh.wpb == 2 || sh.wpb == 4 || sh.wpb == 8) &&
         (sh.qw == 1 || ((sh.qw == 2 || sh.qw == 4) && sh.wpb == sh.qw));
}

int beam_grid(uint32_t d, uint32_t Lmax, uint32_t gw, uint32_t parents, int device, SearchShape sh) {
  if (!beam_shape_ok(sh)) return 0;
  const size_t smem = (size_t)(sh.wpb / sh.qw) * beam_warp_bytes(d, Lmax, beam_cap(gw, parents), sh.hcap);
  if (smem > 227 * 1024) return 0;
  const int t = sh.wpb * 32;
  const int per_sm = sh.qw > 1 ? std::min(BeamKernels<true, false>::blocks_per_sm(t, smem),
                                          BeamKernels<true, true>::blocks_per_sm(t, smem))
                               : std::min(BeamKernels<false, false>::blocks_per_sm(t, smem),
                                          BeamKernels<false, true>::blocks_per_sm(t, smem));
  if (per_sm <= 0) {
    cudaGetLastError();
    return 0;
  }
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  return per_sm * sms;
}

cudaError_t launch_beam(const SearchArgs &a, SearchShape sh, int blocks, cudaStream_t stream) {
  if (!beam_shape_ok(sh)) return cudaErrorInvalidValue;
  SearchArgs b = a;
  b.cap = beam_cap(a.gw, a.parents);
  b.hcap = sh.hcap;
  b.wide_hash = sh.wide ? 1 : 0;
  b.query_warps = sh.qw;
  const size_t smem = (size_t)(sh.wpb / sh.qw) * beam_warp_bytes(b.d, b.Lmax, b.cap, b.hcap);
  const auto launch = sh.qw > 1 ? (b.distinct ? BeamKernels<true, true>::launch : BeamKernels<true, false>::launch)
                                : (b.distinct ? BeamKernels<false, true>::launch : BeamKernels<false, false>::launch);
  launch(blocks, sh.wpb * 32, smem, stream, b);
  return cudaGetLastError();
}

}  // namespace wv

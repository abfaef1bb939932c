// zc_push_exact_det.cu -- the exact build of the push + deposit kernels in
// deterministic mode (zc_push_impl.cuh with DET = true: currents and
// kinetic energy accumulated as 64-bit fixed point).  Compiled with
// --fmad=false, as zc_push_exact.cu.
#include "zc_internal.cuh"
#include "zc_kernels.h"

namespace zc {
namespace exact_det {
#include "zc_push_impl.cuh"
}  // namespace exact_det

cudaError_t launch_push_tiles_exact_det(const PushLaunch &a, cudaStream_t st) {
  return exact_det::launch_push_tiles_variant<true>(a, st);
}

cudaError_t launch_push_spill_exact_det(const PushLaunch &a, int nblocks, cudaStream_t st) {
  return exact_det::launch_push_spill_variant<true>(a, nblocks, st);
}

}  // namespace zc

// zc_push_fast_det.cu -- the fast build of the push + deposit kernels in
// deterministic mode (zc_push_impl.cuh with DET = true: currents and
// kinetic energy accumulated as 64-bit fixed point).  Compiled with the
// flags of zc_push_fast.cu.
#define ZC_FAST 1  // re-associated arithmetic, packed pairs (zc_push_impl.cuh)
#include "zc_internal.cuh"
#include "zc_kernels.h"

namespace zc {
namespace fast_det {
#include "zc_push_impl.cuh"
}  // namespace fast_det

cudaError_t launch_push_tiles_fast_det(const PushLaunch &a, cudaStream_t st) {
  return fast_det::launch_push_tiles_variant<true>(a, st);
}

cudaError_t launch_push_spill_fast_det(const PushLaunch &a, int nblocks, cudaStream_t st) {
  return fast_det::launch_push_spill_variant<true>(a, nblocks, st);
}

}  // namespace zc

// Instantiations of the pencil pass (pencil.cuh) for 1 and 2 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n12(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 1 ? launch_pencil_m<1>(zp, threads, st) : launch_pencil_m<2>(zp, threads, st);
}

}  // namespace crava

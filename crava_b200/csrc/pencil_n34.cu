// Instantiations of the pencil pass (pencil.cuh) for 3 and 4 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n34(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 3 ? launch_pencil_m<3>(zp, threads, st) : launch_pencil_m<4>(zp, threads, st);
}

}  // namespace crava

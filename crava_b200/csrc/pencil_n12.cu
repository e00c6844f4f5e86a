// The pencil pass (pencil.cuh) in its eigen form for 1 and 2 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n12(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 1 ? launch_pencil_z<1, kEig>(zp, threads, st) : launch_pencil_z<2, kEig>(zp, threads, st);
}

}  // namespace crava

// The pencil pass (pencil.cuh) in its eigen form for 3 and 4 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n34(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 3 ? launch_pencil_z<3, kEig>(zp, threads, st) : launch_pencil_z<4, kEig>(zp, threads, st);
}

}  // namespace crava

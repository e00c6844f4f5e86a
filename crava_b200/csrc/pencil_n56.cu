// The pencil pass (pencil.cuh) in its eigen form for 5 and 6 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n56(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 5 ? launch_pencil_z<5, kEig>(zp, threads, st) : launch_pencil_z<6, kEig>(zp, threads, st);
}

}  // namespace crava

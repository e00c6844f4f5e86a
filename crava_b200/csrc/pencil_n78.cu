// The pencil pass (pencil.cuh) in its eigen form for 7 and 8 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n78(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 7 ? launch_pencil_z<7, kEig>(zp, threads, st) : launch_pencil_z<8, kEig>(zp, threads, st);
}

}  // namespace crava

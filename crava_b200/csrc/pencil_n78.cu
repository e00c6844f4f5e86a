// Instantiations of the pencil pass (pencil.cuh) for 7 and 8 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_n78(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 7 ? launch_pencil_m<7>(zp, threads, st) : launch_pencil_m<8>(zp, threads, st);
}

}  // namespace crava

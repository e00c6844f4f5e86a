// The pencil pass (pencil.cuh) in its Cholesky forms for 7 and 8 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_c78(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 7 ? launch_pencil_chol<7>(zp, threads, st) : launch_pencil_chol<8>(zp, threads, st);
}

}  // namespace crava

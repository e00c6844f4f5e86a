// The pencil pass (pencil.cuh) in its Cholesky forms for 1 and 2 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_c12(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 1 ? launch_pencil_chol<1>(zp, threads, st) : launch_pencil_chol<2>(zp, threads, st);
}

}  // namespace crava

// The pencil pass (pencil.cuh) in its Cholesky forms for 3 and 4 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_c34(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 3 ? launch_pencil_chol<3>(zp, threads, st) : launch_pencil_chol<4>(zp, threads, st);
}

}  // namespace crava

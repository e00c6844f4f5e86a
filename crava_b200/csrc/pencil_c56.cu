// The pencil pass (pencil.cuh) in its Cholesky forms for 5 and 6 angle stacks.
#include "pencil.cuh"

namespace crava {

cudaError_t launch_pencil_c56(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.nth == 5 ? launch_pencil_chol<5>(zp, threads, st) : launch_pencil_chol<6>(zp, threads, st);
}

}  // namespace crava

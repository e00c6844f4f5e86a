// Shape and launch of the scalar pencil pass (kernel in zpass.cuh, instantiated by angle count in
// zpass_n12.cu, zpass_n34.cu, zpass_n56.cu and zpass_n78.cu).
#include "zpass.cuh"

namespace crava {

size_t zpass_smem_bytes(int W, int nzp, int nth, int GT, int SB) {
  int G = nth + 3 > 9 ? nth + 3 : 9;
  return sizeof(float2) * ((size_t)nzp + (size_t)(G + GT + 3 * SB) * W * nzp);
}

// The widest tile that fits, with every slot of a phase in one call (GT = G) where it does; 512 threads
// when one CTA fills the SM's shared memory, 256 when two fit.
bool zpass_shape(ZParams& zp, int* threads) {
  const int Gs = std::max(zp.nth + 3, 9);
  const int cand[8][3] = {{4, Gs, 2}, {4, Gs, 1}, {2, Gs, 2}, {2, Gs, 1}, {1, Gs, 2}, {4, 3, 1}, {2, 3, 1}, {1, 3, 1}};
  for (const auto& c : cand) {
    const size_t smem = zpass_smem_bytes(c[0], zp.nzp, zp.nth, c[1], c[2]);
    if (smem > 227 * 1024) continue;
    zp.W = c[0];
    zp.GT = c[1];
    zp.SB = c[2];
    zp.logW = 0;
    while ((1 << zp.logW) < zp.W) zp.logW++;
    zp.nIT = (zp.cnxp + zp.W - 1) / zp.W;
    *threads = smem > 113 * 1024 ? 512 : 256;
    return true;
  }
  return false;
}

cudaError_t launch_zpass(const ZParams& zp, int threads, cudaStream_t st, int* nlaunch) {
  if ((zp.W & (zp.W - 1)) || (1 << zp.logW) != zp.W) return cudaErrorInvalidValue;
  if (3 * zp.SB > zp.GT) return cudaErrorInvalidValue;
  if (nlaunch) (*nlaunch)++;
  switch (zp.nth) {
    case 1: case 2: return launch_zpass_n12(zp, threads, st);
    case 3: case 4: return launch_zpass_n34(zp, threads, st);
    case 5: case 6: return launch_zpass_n56(zp, threads, st);
    case 7: case 8: return launch_zpass_n78(zp, threads, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace crava

// The draws of pair_noise (the pencil pass on pairs) against device_noise3 (the scalar one), bit by bit: every
// bin of an nxp x nyp x nzp block for two realisations.  Prints "<bins> <differing>".
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "zpass.cuh"

using namespace crava;

__global__ void k_check(const __grid_constant__ ZParams P, int i_first, unsigned long long* n) {
  const int pairs = (P.cnxp - i_first + 1) / 2;
  const long long total = 2LL * pairs * P.nyp * P.nzp;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(e & 1);
    const long long r = e >> 1;
    const int i = i_first + 2 * (int)(r % pairs), j = (int)(r / pairs % P.nyp), k = (int)(r / pairs / P.nyp);
    C2 z[3];
    pair_noise(P, s, i, j, k, z);
    for (int u = 0; u < 2; u++) {
      if (i + u < 0 || i + u >= P.cnxp) continue;
      float2 w[3];
      device_noise3(P.seed, s, i + u, j, k, P.nyp, P.nzp, P.cnxp, P.nxp_even != 0, w);
      bool same = true;
      for (int c = 0; c < 3; c++) {
        const float re = u ? z[c].r.y : z[c].r.x, im = u ? z[c].i.y : z[c].i.x;
        same = same && __float_as_uint(re) == __float_as_uint(w[c].x) && __float_as_uint(im) == __float_as_uint(w[c].y);
      }
      atomicAdd(n, 1ull);
      if (!same) atomicAdd(n + 1, 1ull);
    }
  }
}

int main(int argc, char** argv) {
  if (argc < 5) return 2;
  ZParams P;
  std::memset(&P, 0, sizeof P);
  P.nxp = std::atoi(argv[1]);
  P.nyp = std::atoi(argv[2]);
  P.nzp = std::atoi(argv[3]);
  P.cnxp = P.nxp / 2 + 1;
  P.nxp_even = P.nxp % 2 == 0;
  P.seed = 0x9E3779B97F4A7C15ull;
  unsigned long long *d = nullptr, n[2] = {0, 0};
  if (cudaMalloc(&d, sizeof n) != cudaSuccess || cudaMemset(d, 0, sizeof n) != cudaSuccess) return 3;
  k_check<<<256, 128>>>(P, std::atoi(argv[4]), d);
  if (cudaMemcpy(n, d, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
  std::printf("%llu %llu\n", n[0], n[1]);
  return 0;
}

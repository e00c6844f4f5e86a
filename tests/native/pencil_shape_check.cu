// Runs pencil_shape of the built library over every z length, angle count and realisation count that a
// job may have, on narrow and wide blocks, and checks what launch_pencil and the kernel ask of a shape.
// No device is used.  Prints "<shapes> <bad>"; with arguments nxp nyp nzp nth nsim eig, the shape of that job:
// "<W> <SB> <T> <tiles>".
#include <cstdio>
#include <cstdlib>

#include "kernels.cuh"

int main(int argc, char** argv) {
  using namespace crava;
  if (argc > 6) {
    ZParams zp = {};
    zp.nxp = std::atoi(argv[1]);
    zp.cnxp = zp.nxp / 2 + 1;
    zp.nyp = std::atoi(argv[2]);
    zp.nzp = std::atoi(argv[3]);
    zp.nth = std::atoi(argv[4]);
    zp.nsim = std::atoi(argv[5]);
    alignas(16) static float4 table;
    zp.eig = std::atoi(argv[6]) ? &table : nullptr;
    int T = 0;
    if (!pencil_shape(zp, &T)) return 1;
    std::printf("%d %d %d %d\n", zp.W, zp.SB, T, zp.nIT * zp.nyp);
    return 0;
  }
  long shapes = 0, bad = 0;
  for (int nzp = 2; nzp <= 1024; nzp++) {
    int m = nzp;
    for (int p : {2, 3, 5, 7})
      while (m % p == 0) m /= p;
    if (m != 1) continue;
    for (int nth = 1; nth <= kMaxTheta; nth++) {
      for (int nsim = 0; nsim <= kMaxSim; nsim++)
        for (int side : {2, 31, 540, 4096}) {
          ZParams zp = {};
          zp.nxp = zp.nyp = side;
          zp.cnxp = side / 2 + 1;
          zp.nzp = nzp;
          zp.nth = nth;
          zp.nsim = nsim;
          int T = 0;
          shapes++;
          const bool ok = pencil_shape(zp, &T) && T >= 64 && T <= 512 && T % 32 == 0 && zp.W == 2 * zp.NP &&
                          (1 << zp.logNP) == zp.NP && zp.SB >= (nsim ? 1 : 0) && zp.SB <= 4 &&
                          nzp * zp.NP <= 16 * T && pencil_smem_bytes(zp.W, nzp, nth, zp.SB) + 64 <= 227 * 1024;
          if (!ok && bad++ < 10) std::fprintf(stderr, "nzp %d nth %d nsim %d side %d: W %d SB %d T %d\n", nzp, nth, nsim, side, zp.W, zp.SB, T);
        }
    }
  }
  std::printf("%ld %ld\n", shapes, bad);
  return 0;
}

// Plan, tile shape and launch of the pencil pass (kernel in pencil.cuh, instantiated by angle
// count in pencil_n*.cu and pencil_c*.cu).
#include "pencil.cuh"

#include <algorithm>

namespace crava {

namespace {

// n as a product of `left` radices, none above `top`, descending; the first found has the largest
// leading radix, which the last (storing) inverse stage takes
bool split(int n, int left, int top, int8_t* out) {
  static const int radices[] = {
#define CRAVA_CASE(RR) RR,
      CRAVA_Z_RADICES(CRAVA_CASE)
#undef CRAVA_CASE
  };
  constexpr int nr = sizeof(radices) / sizeof(radices[0]);
  if (left == 0) return n == 1;
  for (int i = nr - 1; i >= 0; i--) {
    const int r = radices[i];
    if (r > top || n % r) continue;
    out[0] = (int8_t)r;
    if (split(n / r, left - 1, r, out + 1)) return true;
  }
  return false;
}

}  // namespace

// The fewest stages (each costs a round trip through shared memory and a barrier), then the
// smallest largest radix (registers, and more items per stage): 256 = 16 x 16, 200 = 20 x 10,
// 125 = 5 x 5 x 5.
bool pencil_plan(int n, ZPlan& z) {
  z.n = n;
  for (z.ns = 1; z.ns <= 10; z.ns++)
    for (int top = 2; top <= 20; top++)
      if (split(n, z.ns, top, z.radix)) return true;
  return false;
}

int pencil_kz(const ZPlan& z, int p) {
  int kz = 0, mul = 1, len = z.n;
  for (int s = 0; s < z.ns; s++) {
    len /= z.radix[s];
    kz += mul * (p / len);
    p %= len;
    mul *= z.radix[s];
  }
  return kz;
}

static int tile_slot(int nth, int SB) { return std::max(nth + 3, 6 + 3 * SB); }

static int tile_ps(int W, int nth, int SB) {
  const int NP = W / 2, D = tile_slot(nth, SB);
  int words = D * NP + NP + (NP + 1) / 2;
  // an odd number of 16-byte words puts the positions of neighbouring threads on different banks;
  // two pairs want 2 mod 4
  if (NP == 1 && words % 2 == 0) words++;
  if (NP == 2 && words % 4 == 1) words++;
  return 16 * words;
}

size_t pencil_smem_bytes(int W, int nzp, int nth, int SB) {
  return 8 * (size_t)even_up_z(nzp) + 96 + 2 * (size_t)((nzp + 7) & ~7) + (size_t)tile_ps(W, nth, SB) * nzp;
}

// CTAs whose tiles of `smem` bytes share an SM: 228 KB, of which each takes 1 KB and its static shared
// memory (64 bytes at most) besides, in units of 128 bytes.  A tile at the cap of 227 KB is one.
constexpr size_t kStaticSmem = 64;
static int tiles_per_sm(size_t smem) {
  return std::max(1, (int)(228 * 1024 / ((smem + kStaticSmem + 127) / 128 * 128 + 1024)));
}
// ... and at T threads (128 registers each).
static int resident(size_t smem, int T) { return std::max(1, std::min(tiles_per_sm(smem), 512 / T)); }

// The tile.  Two or more CTAs of 128..256 threads on an SM overlap one's copies and barriers with the
// other's arithmetic (270x270x256, 5 angles, 4 realisations: W 8, 512 threads 1.30 ms; W 4, two of
// 256 1.25), so a shape that allows it is preferred; then the wider tile (longer rows in global
// memory) and the larger realisation batch (an inverse stage of SB realisations keeps 6 SB / R of the
// threads busy).  Relative costs as measured at 64 to 320 points, 1 to 16 realisations; a shape
// whose tiles fill the last wave badly pays for it (64x64x128: W 8 39 us, W 4 31).
bool pencil_shape(ZParams& zp, int* threads) {
  const size_t cap = 227 * 1024 - kStaticSmem;
  const int key = zp.nzp * 16 + zp.nth, least = zp.nsim ? 1 : 0, most = std::min(zp.nsim, 4);
  const int per = zp.eig ? 2 : 1;       // bins per thread of the per-bin step
  if (!pencil_plan(zp.nzp, zp.z)) return false;
  const int tw = tuned("pencil_w", key, 0), ts = tuned("pencil_sb", key, -1), tt = tuned("pencil_threads", key, 0);
  int W = 0, SB = 0, T = 0;
  double cost = 1e30;
  for (int w = 8; w >= 2; w /= 2) {
    if (tw > 0 && w > std::max(2, tw)) continue;
    if (tw > 0 && W) break;             // the schedule's width, or the widest below it that fits
    for (int b = 4; b >= least; b--) {
      if (b > most || (b == 3 && most != 3 && ts != 3)) continue;
      if (ts >= 0 && b > std::max(least, std::min(most, ts))) continue;
      const size_t smem = pencil_smem_bytes(w, zp.nzp, zp.nth, b);
      if (smem > cap) continue;
      const int fit = std::min(4, tiles_per_sm(smem));
      int t = fit >= 2 ? 512 / fit / 32 * 32 : 512;
      t = std::max(64, std::min(t, (zp.nzp * w / per + 31) / 32 * 32));
      const int ctas = resident(smem, t);
      const long long tiles = (long long)((zp.cnxp + w - 1) / w) * zp.nyp, slots = 148LL * ctas;
      // eight bins only where they leave two tiles for every SM: a small block is as fast as one tile, and half
      // as wide a tile is faster (20x20x40, 2 angles, 16 realisations, 40 tiles of 8 bins: 105 us, 60 of 4: 54)
      if (w == 8 && tw <= 0 && tiles < 2 * 148) break;
      const double fill = (double)tiles / ((tiles + slots - 1) / slots * slots);
      double c = w == 8 ? 1.0 : w == 4 ? 1.02 : 1.35;
      if (zp.nsim > 1) c *= b == 1 ? 1.05 : b == 4 && w == 8 ? 1.03 : 1.0;
      if (zp.nsim > 1 && w == 4) c *= b == 1 ? 1.12 : b == 4 ? 1.01 : 1.05;
      if (ctas < 2) c *= 1.15;
      c /= 0.5 + 0.5 * fill;
      if (c < cost) {
        cost = c;
        W = w;
        SB = b;
        T = t;
      }
      if (ts >= 0) break;
    }
  }
  if (!W) return false;
  zp.W = W;
  zp.NP = W / 2;
  zp.logNP = 0;
  while ((1 << zp.logNP) < zp.NP) zp.logNP++;
  // every pair one 16-byte access: the z stride an even number of bins, every grid 16-byte aligned
  uintptr_t a = 8 * ((uintptr_t)zp.nyp * zp.cnxp);
  for (int l = 0; l < zp.nth; l++) a |= (uintptr_t)zp.data[l];
  for (int c = 0; c < 3; c++) a |= (uintptr_t)zp.mean[c];
  for (int c = 0; c < 6; c++) a |= (uintptr_t)zp.cov[c];
  for (int c = 0; c < 3 * zp.nsim; c++) a |= (uintptr_t)zp.sim[c];
  zp.vec = a % 16 == 0;
  zp.nIT = (zp.cnxp + zp.vec + W - 1) / W;
  zp.SB = SB;
  zp.D = tile_slot(zp.nth, SB);
  zp.PS = tile_ps(W, zp.nth, SB);
  zp.swz = zp.NP == 4 && zp.nzp % 4 == 0;
  const int items = zp.nzp * zp.NP;
  // A block whose tiles are all resident at once: a tile's time is its rounds of pairs (of bins in the Cholesky
  // forms, each as long as a factorisation) and of transform items, so the threads of an SM go to the r tiles that it
  // gets where that saves a round (24x36x42, 8 realisations, 144 tiles: the job 60.6 us at 96 threads, 46.5 at 192;
  // 24x24x128: 62.9 at 256, 53.8 at 384; 48x50x72, 6 angles, FP64, 350 tiles of 288 bins: the pass 96 -> 70 us at 160
  // instead of 128).  Not so many that some tiles wait (48x48x48, 336 tiles: 80.3 at 128, 103.6 at 192).
  const long long tiles = (long long)zp.nIT * zp.nyp;
  const int fit = std::min(4, tiles_per_sm(pencil_smem_bytes(W, zp.nzp, zp.nth, SB)));
  if (tiles <= 148LL * fit) {
    const int lines = std::max(3 * SB, std::max(zp.nth + 3, 8)) * zp.NP;
    const int work = std::max(zp.nzp * W / per, lines * (zp.nzp / zp.z.radix[zp.z.ns - 1]));
    int least = 1 << 30;
    for (int r = fit; r >= (int)((tiles + 147) / 148); r--) {
      const int t = std::max(64, std::min(512 / r / 32 * 32, (work + 31) / 32 * 32));
      const int rounds = (work + t - 1) / t;
      if (rounds < least) {
        least = rounds;
        T = t;
      }
    }
  }
  if (tt > 0) T = std::max(64, std::min(512, tt / 32 * 32));
  // two bits per item of a thread hold the failed factorisations: at most 16 items each
  T = std::max(T, std::min(512, (items / 16 + 31) / 32 * 32));
  *threads = T;
  return true;
}

cudaError_t launch_pencil(const ZParams& zp, int threads, cudaStream_t st, int* nlaunch) {
  if (zp.NP < 1 || zp.W != 2 * zp.NP || (1 << zp.logNP) != zp.NP || threads < 64 || threads > 512 ||
      zp.SB < (zp.nsim ? 1 : 0) || zp.SB > 4 || zp.nzp * zp.NP > 16 * threads ||
      (zp.keep_resid && !z_inlined(zp.nzp)))
    return cudaErrorInvalidValue;
  if (nlaunch) (*nlaunch)++;
  const bool chol = zp.fp64_threshold > 0.f || !zp.eig;
  switch (zp.nth) {
    case 1: case 2: return chol ? launch_pencil_c12(zp, threads, st) : launch_pencil_n12(zp, threads, st);
    case 3: case 4: return chol ? launch_pencil_c34(zp, threads, st) : launch_pencil_n34(zp, threads, st);
    case 5: case 6: return chol ? launch_pencil_c56(zp, threads, st) : launch_pencil_n56(zp, threads, st);
    case 7: case 8: return chol ? launch_pencil_c78(zp, threads, st) : launch_pencil_n78(zp, threads, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace crava

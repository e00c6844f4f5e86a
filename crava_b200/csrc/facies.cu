// Facies probabilities from the posterior elastic parameters (sm_100a).
//
//   k_facies_prob_corners  per voxel: trilinear lookup of every facies density volume at the
//                   posterior (ln Vp, ln Vs, ln rho), prior-weighted, normalised with the
//                   undefined-facies floor (FaciesProb::calculateFaciesProb and findDensity,
//                   src/faciesprob.cpp:1909-2075, 1307-1423), with local noise over 2^nang
//                   corner volumes weighted by the trace's relative noise scales
//   k_facies_pack   the density volumes repacked facies-interleaved for those lookups
//   k_smoother_*    the normalised Gaussian smoother of the facies histograms
//   k_spec_mul      spectrum product for the Gaussian smoothing of the facies histograms
//                   (FaciesProb::makeFaciesDens, src/faciesprob.cpp:440-522)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "facies.cuh"

namespace crava {

template <bool PAIRS>
__global__ void k_facies_prob_corners(const float* __restrict__ vp, const float* __restrict__ vs,
                                      const float* __restrict__ rho, int nx, int ny, int nz, int rnxp_in, int nyp_in,
                                      int rnxp_out, const __grid_constant__ FaciesCorners C, int nf, FaciesPrior pr,
                                      float undef_sum, FaciesOut out, float* __restrict__ seis_lh) {
  // One voxel a thread and round, across the row ends: a voxel costs several hundred instructions, so that rows by whole
  // warps pay for their idle lanes (37x400x60, 6 facies, 20x20x10 bins: 68 -> 53 us; 270x270x256 797 -> 745) and two
  // 32-bit divisions do not show.  k_facies_prob_single, a few times cheaper, takes rows.
  const size_t n = (size_t)rnxp_out * ny * nz;
  const bool word = n <= 0xffffffffu;      // 32-bit divisions
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const size_t r = word ? (size_t)((unsigned)e / (unsigned)rnxp_out) : e / rnxp_out;
    const int i = (int)(e - r * rnxp_out), k = (int)(word ? (unsigned)r / (unsigned)ny : r / ny);
    const int j = (int)(r - (size_t)k * ny);
    if (i >= nx) {
      for (int f = 0; f <= nf; f++) out.p[f][e] = kRMissing;
      if (seis_lh) seis_lh[e] = kRMissing;
      continue;
    }
    const size_t g = i + (size_t)rnxp_in * ((size_t)j + (size_t)nyp_in * k);
    const float v[3] = {vp[g], vs[g], rho[g]};
    float val[kMaxFacies];
    const float sum = facies_voxel<PAIRS>(v, i, j, nx, ny, C, nf, pr, undef_sum, val);
    for (int f = 0; f < nf; f++) out.p[f][e] = val[f] / sum;
    out.p[nf][e] = undef_sum / sum;
    if (seis_lh) seis_lh[e] = sum;
  }
}

// The same for one volume (no local noise) of at most four facies, the usual case, with everything in
// registers: the general form keeps its facies in local memory and spends 562 instructions a voxel.
// 270x270x256, 3 facies, 100x100x50 bins, with the packing: 0.66 -> 0.37 ms.
struct FaciesSingle {
  const float4* dens;
  int nb[3];
  double vmin[3], dv[3];
};
template <bool PAIRS>
__global__ void __launch_bounds__(256) k_facies_prob_single(const float* __restrict__ vp, const float* __restrict__ vs,
                                                            const float* __restrict__ rho, int nx, int ny, int nz,
                                                            int rnxp_in, int nyp_in, int rnxp_out,
                                                            const __grid_constant__ FaciesSingle C, int nf,
                                                            const __grid_constant__ FaciesPrior pr, float undef_sum,
                                                            const __grid_constant__ FaciesOut out,
                                                            float* __restrict__ seis_lh) {
  const int rows = ny * nz;
  const int sk = C.nb[0], sl = C.nb[0] * C.nb[1];
  for (int r = blockIdx.x * blockDim.y + threadIdx.y; r < rows; r += gridDim.x * blockDim.y) {
    const int k = r / ny, j = r - k * ny;
    const size_t e0 = (size_t)rnxp_out * r, g0 = (size_t)rnxp_in * ((size_t)j + (size_t)nyp_in * k);
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < rnxp_out; i += gridDim.y * blockDim.x) {
      const size_t e = e0 + i;
      if (i >= nx) {
        for (int f = 0; f <= nf; f++) out.p[f][e] = kRMissing;
        if (seis_lh) seis_lh[e] = kRMissing;
        continue;
      }
      int a1, a2, b1, b2, c1, c2;
      float wj, wk, wl;
      axis_weights(__ldg(vp + g0 + i), C.vmin[0], C.dv[0], C.nb[0], a1, a2, wj);
      axis_weights(__ldg(vs + g0 + i), C.vmin[1], C.dv[1], C.nb[1], b1, b2, wk);
      axis_weights(__ldg(rho + g0 + i), C.vmin[2], C.dv[2], C.nb[2], c1, c2, wl);
      const float uj = 1.0f - wj, uk = 1.0f - wk, ul = 1.0f - wl;
      const float w8[8] = {uj * uk * ul, uj * uk * wl, uj * wk * ul, uj * wk * wl,
                           wj * uk * ul, wj * uk * wl, wj * wk * ul, wj * wk * wl};
      const int cell[4] = {a1 + sk * b1 + sl * c1, a1 + sk * b1 + sl * c2, a1 + sk * b2 + sl * c1, a1 + sk * b2 + sl * c2};
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if constexpr (PAIRS) {
          ldg_pair(C.dens + 2 * (size_t)cell[q], x[q], x[4 + q]);
          if (a1 == a2) x[4 + q] = x[q];
        } else {
          x[q] = __ldg(C.dens + cell[q]);
          x[4 + q] = __ldg(C.dens + cell[q] + (a2 - a1));
        }
      }
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        d[0] += w8[q] * x[q].x;
        d[1] += w8[q] * x[q].y;
        d[2] += w8[q] * x[q].z;
        d[3] += w8[q] * x[q].w;
      }
      float sum = undef_sum;
#pragma unroll
      for (int f = 0; f < 4; f++) {
        d[f] = f < nf ? pr.p[f] * (d[f] > 0.f ? d[f] : 0.f) : 0.f;
        if (f < nf) sum += d[f];
      }
#pragma unroll
      for (int f = 0; f < 4; f++)
        if (f < nf) out.p[f][e] = d[f] / sum;
      out.p[nf][e] = undef_sum / sum;
      if (seis_lh) seis_lh[e] = sum;
    }
  }
}

// Packs one density volume: cell (j, k, l) <- the nf facies values max(0, dens_f) of (j, k, l) and, in pairs,
// of (j + 1, k, l) (the last bin's own again), four per float4 (zero beyond nf), the pair of a group of
// four side by side; dens_f at src + f * fstride + j + rs (k + nb1 l).
template <bool PAIRS>
__global__ void k_facies_pack(const float* __restrict__ src, int nb0, int nb1, int nb2, int rs, size_t fstride,
                              int nf, float4* __restrict__ dst) {
  const int nf4 = (nf + 3) / 4;
  const size_t ncell = (size_t)nb0 * nb1 * nb2;
  for (size_t cidx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; cidx < ncell * nf4;
       cidx += (size_t)gridDim.x * blockDim.x) {
    const size_t cell = cidx / nf4;
    const int g = (int)(cidx % nf4);
    const int j = (int)(cell % nb0);
    const size_t kl = cell / nb0;
    const int kk = (int)(kl % nb1), l = (int)(kl / nb1);
    const size_t o = (size_t)rs * ((size_t)kk + (size_t)nb1 * l);
#pragma unroll
    for (int h = 0; h < (PAIRS ? 2 : 1); h++) {
      const int jh = min(j + h, nb0 - 1);
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int f = 4 * g + u;
        x[u] = f < nf ? fmaxf(0.f, __ldg(src + fstride * f + o + jh)) : 0.f;
      }
      dst[(PAIRS ? 2 : 1) * cidx + h] = make_float4(x[0], x[1], x[2], x[3]);
    }
  }
}

// ------------------------------------------------------------------ the Gaussian smoother
//
// FaciesProb::makeFaciesDens (src/faciesprob.cpp:447-496): exp(-factor / 2) over cyclic bin offsets,
// normalised by its sum, which the reference accumulates in a float, in bin order.  That sum
// loses the tails (2.7e-4 of it at 100x100x50 bins), so its order is part of the result: the values are formed in
// parallel, and one CTA adds them in order, chunk by chunk, keeping only those that can change the sum
// (v < ulp(sum) / 2 leaves it as it is).  exp is the double function rounded to float, which equals
// a correctly rounded expf.  The host loops it replaces took 3.5 ms a call.
struct Smoother {
  int na, nb, nr, rna;
  double dv[3], S[6];          // S: 00 11 22 10 20 21
};

__global__ void k_smoother_fill(const __grid_constant__ Smoother P, float* __restrict__ g) {
  const size_t n = (size_t)P.rna * P.nb * P.nr;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(e % P.rna);
    const size_t kl = e / P.rna;
    const int k = (int)(kl % P.nb), l = (int)(kl / P.nb);
    if (j >= P.na) {
      g[e] = 0.f;
      continue;
    }
    const int ji = j <= P.na / 2 ? j : j - P.na, ki = k <= P.nb / 2 ? k : k - P.nb, li = l <= P.nr / 2 ? l : l - P.nr;
    auto term = [](int two_a, double da, int b, double db, double s) {
      return __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn((double)two_a, da), (double)b), db), s);
    };
    double f = term(ji, P.dv[0], ji, P.dv[0], P.S[0]);
    f = __dadd_rn(f, term(ki, P.dv[1], ki, P.dv[1], P.S[1]));
    f = __dadd_rn(f, term(li, P.dv[2], li, P.dv[2], P.S[2]));
    f = __dadd_rn(f, term(2 * ji, P.dv[0], ki, P.dv[1], P.S[3]));
    f = __dadd_rn(f, term(2 * ji, P.dv[0], li, P.dv[2], P.S[4]));
    f = __dadd_rn(f, term(2 * ki, P.dv[1], li, P.dv[2], P.S[5]));
    g[e] = (float)exp((double)__fmul_rn(-0.5f, (float)f));
  }
}

constexpr int kSumThreads = 1024, kSumPer = 8, kSumChunk = kSumThreads * kSumPer;

// *out = the float sum of the na x nb x nr values of g (rows of rna) in order
__global__ void __launch_bounds__(kSumThreads) k_smoother_sum(const float* __restrict__ g, int na, int rna, long long n,
                                                              float* __restrict__ out) {
  __shared__ float kept[kSumChunk];
  __shared__ int warp_n[32];
  __shared__ float sum_s;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) sum_s = 0.f;
  __syncthreads();
  for (long long c0 = 0; c0 < n; c0 += kSumChunk) {
    const float s0 = sum_s;
    const float half = 0.5f * (__uint_as_float(__float_as_uint(s0) + 1u) - s0);
    float v[kSumPer];
    int m = 0;
#pragma unroll
    for (int u = 0; u < kSumPer; u++) {
      const long long e = c0 + tid * kSumPer + u;
      float x = 0.f;
      if (e < n) {
        const long long row = e / na;
        x = __ldg(g + row * rna + (e - row * na));
      }
      if (x != 0.f && !(x < half)) v[m++] = x;
    }
    // stable compaction: exclusive prefix of the threads' counts
    int p = m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, p, d);
      if (lane >= d) p += y;
    }
    if (lane == 31) warp_n[wid] = p;
    __syncthreads();
    if (wid == 0) {
      int w = warp_n[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += y;
      }
      warp_n[lane] = w;
    }
    __syncthreads();
    const int o = p - m + (wid ? warp_n[wid - 1] : 0), total = warp_n[31];
    for (int u = 0; u < m; u++) kept[o + u] = v[u];
    __syncthreads();
    if (tid == 0) {
      float s = s0;
      int u = 0;
      for (; u + 8 <= total; u += 8) {
        float x[8];
#pragma unroll
        for (int w = 0; w < 8; w++) x[w] = kept[u + w];
#pragma unroll
        for (int w = 0; w < 8; w++) s = __fadd_rn(s, x[w]);
      }
      for (; u < total; u++) s = __fadd_rn(s, kept[u]);
      sum_s = s;
    }
    __syncthreads();
  }
  if (tid == 0) *out = sum_s;
}

__global__ void k_smoother_scale(float* __restrict__ g, size_t n, const float* __restrict__ sum) {
  const float s = *sum;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    g[e] = __fdiv_rn(g[e], s);
}

// The normalised smoother of na x nb x nr bins in FFTGrid layout (rows of 2 (na / 2 + 1)); S = sigma_inv
// (3 x 3); sum: one float of scratch.
cudaError_t launch_facies_smoother(float* g, float* sum, int na, int nb, int nr, const double* dv, const double* S,
                                   cudaStream_t st, int* nlaunch) {
  Smoother P;
  P.na = na;
  P.nb = nb;
  P.nr = nr;
  P.rna = 2 * (na / 2 + 1);
  for (int d = 0; d < 3; d++) P.dv[d] = dv[d];
  P.S[0] = S[0]; P.S[1] = S[4]; P.S[2] = S[8]; P.S[3] = S[3]; P.S[4] = S[6]; P.S[5] = S[7];
  const size_t n = (size_t)P.rna * nb * nr;
  const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 8);
  k_smoother_fill<<<blocks, 256, 0, st>>>(P, g);
  k_smoother_sum<<<1, kSumThreads, 0, st>>>(g, na, P.rna, (long long)na * nb * nr, sum);
  k_smoother_scale<<<blocks, 256, 0, st>>>(g, n, sum);
  if (nlaunch) *nlaunch += 3;
  return cudaGetLastError();
}

// a <- a * b (complex) over n bins
__global__ void k_spec_mul(float2* __restrict__ a, const float2* __restrict__ b, size_t n) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    float2 x = a[e], y = b[e];
    a[e] = make_float2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
  }
}

cudaError_t launch_facies_prob_corners(const float* vp, const float* vs, const float* rho, int nx, int ny, int nz,
                                       int rnxp_in, int nyp_in, int rnxp_out, const FaciesCornersHost& hc, int nf,
                                       const float* prior, float undef_sum, float* const* out, float* seis_lh,
                                       cudaStream_t st) {
  if (nf < 1 || nf > kMaxFacies || hc.nang < 0 || hc.nang > kMaxFaciesAngles) return cudaErrorInvalidValue;
  cudaError_t e = launch_facies_pack(hc, nf, st);
  if (e != cudaSuccess) return e;
  return launch_facies_eval(vp, vs, rho, nx, ny, nz, rnxp_in, nyp_in, rnxp_out, hc, nf, prior, undef_sum, out, seis_lh,
                            st);
}

cudaError_t launch_facies_eval(const float* vp, const float* vs, const float* rho, int nx, int ny, int nz, int rnxp_in,
                               int nyp_in, int rnxp_out, const FaciesCornersHost& hc, int nf, const float* prior,
                               float undef_sum, float* const* out, float* seis_lh, cudaStream_t st) {
  if (nf < 1 || nf > kMaxFacies || hc.nang < 0 || hc.nang > kMaxFaciesAngles) return cudaErrorInvalidValue;
  FaciesPrior pr;
  FaciesOut po;
  for (int f = 0; f < nf; f++) pr.p[f] = prior[f];
  for (int f = 0; f <= nf; f++) po.p[f] = out[f];
  const FaciesCorners C = facies_corners(hc);
  if (hc.nang == 0 && nf <= 4 && (size_t)hc.box[0].nb[0] * hc.box[0].nb[1] * hc.box[0].nb[2] < (1u << 30)) {
    // a few long rows (a section of 4000 traces has 2 per slice) are shared by several warps each, until eight CTAs an
    // SM have work
    dim3 blocks((unsigned)std::min<size_t>(((size_t)ny * nz + 7) / 8, 148 * 32));
    blocks.y = (unsigned)std::max(1, std::min((rnxp_out + 31) / 32, (148 * 8 + (int)blocks.x - 1) / (int)blocks.x));
    FaciesSingle F;
    F.dens = hc.packed[0];
    for (int d = 0; d < 3; d++) {
      F.nb[d] = hc.box[0].nb[d];
      F.vmin[d] = hc.box[0].vmin[d];
      F.dv[d] = hc.box[0].dv[d];
    }
    (hc.pairs ? k_facies_prob_single<true> : k_facies_prob_single<false>)<<<blocks, dim3(32, 8), 0, st>>>(
        vp, vs, rho, nx, ny, nz, rnxp_in, nyp_in, rnxp_out, F, nf, pr, undef_sum, po, seis_lh);
    return cudaGetLastError();
  }
  const int flat = (int)std::min<size_t>(((size_t)rnxp_out * ny * nz + 255) / 256, 148 * 32);
  (hc.pairs ? k_facies_prob_corners<true> : k_facies_prob_corners<false>)<<<flat, 256, 0, st>>>(
      vp, vs, rho, nx, ny, nz, rnxp_in, nyp_in, rnxp_out, C, nf, pr, undef_sum, po, seis_lh);
  return cudaGetLastError();
}

cudaError_t launch_facies_pack(const FaciesCornersHost& hc, int nf, cudaStream_t st) {
  if (nf < 1 || nf > kMaxFacies || hc.nang < 0 || hc.nang > kMaxFaciesAngles) return cudaErrorInvalidValue;
  const int nf4 = (nf + 3) / 4;
  for (int c = 0; c < (1 << hc.nang); c++) {
    const size_t units = (size_t)hc.box[c].nb[0] * hc.box[c].nb[1] * hc.box[c].nb[2] * nf4;
    const int pb = (int)std::min<size_t>((units + 255) / 256, 148 * 8);
    (hc.pairs ? k_facies_pack<true> : k_facies_pack<false>)<<<pb, 256, 0, st>>>(
        hc.dens[c], hc.box[c].nb[0], hc.box[c].nb[1], hc.box[c].nb[2], hc.box[c].rs, hc.box[c].fstride, nf, hc.packed[c]);
  }
  return cudaGetLastError();
}

FaciesCorners facies_corners(const FaciesCornersHost& hc) {
  FaciesCorners C;
  C.nang = hc.nang;
  C.pairs = hc.pairs;
  C.t = hc.t;
  for (int c = 0; c < (1 << hc.nang); c++) {
    for (int d = 0; d < 3; d++) {
      C.box[c].nb[d] = hc.box[c].nb[d];
      C.box[c].vmin[d] = hc.box[c].vmin[d];
      C.box[c].dv[d] = hc.box[c].dv[d];
    }
    C.box[c].rs = hc.box[c].rs;
    C.box[c].fstride = hc.box[c].fstride;
    C.dens[c] = hc.packed[c];
  }
  return C;
}

size_t facies_packed_bytes(const FaciesBoxHost& b, int nf, bool pairs) {
  return (pairs ? 2 : 1) * sizeof(float4) * (size_t)b.nb[0] * b.nb[1] * b.nb[2] * ((nf + 3) / 4);
}

// Above 8 MB, where scattered cells are fetched from the L2, and up to 256 MB, twice what it holds (facies.cuh has both
// sides).
bool facies_pairs(const FaciesCornersHost& hc, int nf) {
  size_t bytes = 0;
  for (int c = 0; c < (1 << hc.nang); c++) bytes += facies_packed_bytes(hc.box[c], nf, true);
  return bytes > 8u << 20 && bytes <= 256u << 20;
}

cudaError_t launch_spec_mul(float2* a, const float2* b, size_t n, cudaStream_t st) {
  int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
  k_spec_mul<<<blocks, 256, 0, st>>>(a, b, n);
  return cudaGetLastError();
}

}  // namespace crava

// The inverse x transform of the three posterior-mean grids with the facies probabilities
// evaluated in the same pass (sm_100a): the rows of the three grids go through the c2r
// transform of k_xc2r4 (written back as the real posterior mean, the FFTGrid::invFFTInPlace
// output), stay in shared memory, and every voxel of those rows is evaluated there by
// facies_voxel (FaciesProb::calculateFaciesProb, src/faciesprob.cpp:1909-2075), so the
// posterior mean is not read back from memory for the facies pass.
#pragma once
#include "facies.cuh"
#include "fft4.cuh"

namespace crava {

// rows r = j + nyp k of rpc-row chunks; shared: twiddle tables, the rows of the three grids (buffers of
// bw float2), the exchange rows Z of the lengths that are not taken in pairs
template <int N1, int N2>
__global__ void __launch_bounds__(256) k_xc2r4_facies(const __grid_constant__ FaciesFuse F,
                                                      const __grid_constant__ FaciesCorners C, int rows, int rpc, int bw,
                                                      const float2* __restrict__ twg, const float2* __restrict__ twn) {
  constexpr int H = N1 * N2, CN = H + 1;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  float2* twh = tw + H;
  float2* V = twh + H;
  const int row0 = blockIdx.x * rpc, nr = min(rpc, rows - row0);
  for (int t = threadIdx.x; t < H; t += blockDim.x) {
    tw[t] = twg[t];
    twh[t] = twn[t];
  }
  for (int a = 0; a < 3; a++) rows_in(V + a * bw, reinterpret_cast<const float2*>(F.mean[a]) + (size_t)row0 * CN, nr * CN, 8);
  cp_async_wait_0();
  __syncthreads();
  for (int a = 0; a < 3; a++) {
    float2* B = V + a * bw;
    if constexpr (RowPairs<N1, N2>::ok) xc2r4_pairs<N1, N2>(B, nr, F.scale, tw, twh);
    else xc2r4_staged<N1, N2>(B, B, nr, F.scale, tw, twh, V + 3 * bw);
    rows_out(reinterpret_cast<float2*>(F.mean[a]) + (size_t)row0 * CN, B, nr * CN, 8);
    __syncthreads();
  }
  const float* Vf = reinterpret_cast<const float*>(V);
  for (int e = threadIdx.x; e < nr * F.rnxp_out; e += blockDim.x) {
    const int r = e / F.rnxp_out, i = e - r * F.rnxp_out;
    const int row = row0 + r, k = row / F.nyp, j = row - k * F.nyp;
    if (j >= F.ny || k >= F.nz) continue;
    const size_t o = (size_t)i + (size_t)F.rnxp_out * ((size_t)j + (size_t)F.ny * k);
    if (i >= F.nx) {
      for (int f = 0; f <= F.nf; f++) F.out.p[f][o] = kRMissing;
      if (F.seis_lh) F.seis_lh[o] = kRMissing;
      continue;
    }
    const int s = 2 * r * CN + i;   // sample i of row r in a grid's buffer of 2 bw floats
    const float v[3] = {Vf[s], Vf[2 * bw + s], Vf[4 * bw + s]};
    float val[kMaxFacies];
    const float sum = C.pairs ? facies_voxel<true>(v, i, j, F.nx, F.ny, C, F.nf, F.pr, F.undef_sum, val)
                              : facies_voxel<false>(v, i, j, F.nx, F.ny, C, F.nf, F.pr, F.undef_sum, val);
    for (int f = 0; f < F.nf; f++) F.out.p[f][o] = val[f] / sum;
    F.out.p[F.nf][o] = F.undef_sum / sum;
    if (F.seis_lh) F.seis_lh[o] = sum;
  }
}

// threads per CTA: schedule key x4_facies_threads (n = h), default 128; rows per CTA by the row kernel's
// items
template <int N1, int N2>
static cudaError_t x4_facies(const FaciesFuse& F, const FaciesCorners& C, int rows, const float2* tw,
                             const float2* twn, cudaStream_t st) {
  using L = RowLayout<N1, N2>;
  const int T = std::max(32, std::min(256, tuned("x4_facies_threads", L::H, 128) / 32 * 32));
  const int np = std::max(1, T / N1 / 2), rpc = RowPairs<N1, N2>::ok ? 2 * np : std::max(1, T / N1);
  const int bw = RowPairs<N1, N2>::ok ? RowPairs<N1, N2>::words(np) : even_up(rpc * (L::H + 1));
  const int Tp = RowPairs<N1, N2>::ok ? std::max(T, (np * N1 + 31) / 32 * 32) : T;
  const size_t smem = sizeof(float2) * (2 * (size_t)L::H + 3 * (size_t)bw + (RowPairs<N1, N2>::ok ? 0 : (size_t)rpc * L::PITCH));
  cudaError_t e = cudaFuncSetAttribute(k_xc2r4_facies<N1, N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_xc2r4_facies<N1, N2><<<(unsigned)((rows + rpc - 1) / rpc), Tp, smem, st>>>(F, C, rows, rpc, bw, tw, twn);
  return cudaGetLastError();
}

}  // namespace crava

// The pencil pass of jobs that keep their residual spectra, at the z lengths without an inlined split
// (sm_100a): the same pass as pencil.cuh with the scalar Stockham transforms (fft_core.cuh) in z.
//
// The residuals d - K mu_post are differences: every bin carries the FP32 rounding of the large
// constant background (ln 3000) through the transforms and K mu, 5e-5 of the residuals, so another
// order of the forward transforms' roundings, however exact, changes them by that much.  For these jobs
// the forward transforms keep the order they had (GridSet.plain for x and y), and this kernel
// keeps it in z; at 128, 256 and 320 points pencil.cuh has the same splits and agrees to 1e-6.
// (Timings beside pencil.cuh: 250x250x200, 5 angles, 4 realisations 2.21 against 1.28 ms.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fft_core.cuh"
#include "kernels.cuh"
#include "pencil_bin.cuh"
#include "pencil_common.cuh"

namespace crava {

// Box-Muller with the hardware approximations of log, sine and cosine: their absolute
// errors (about 2^-21 on these ranges) are far below what the normals' statistics can show.
// u1 from a 26-bit integer a (radius: the largest |normal| is sqrt(2 ln 2^27) = 6.1), the angle
// from a 16-bit integer b (resolution 2 pi / 65536).
__device__ __forceinline__ void box_muller(uint32_t a, uint32_t b, float& n0, float& n1) {
  float u1 = ((float)a + 0.5f) * 1.4901161193847656e-08f;        // (a + 1/2) / 2^26, in (0, 1)
  float u2 = ((float)b + 0.5f) * 1.52587890625e-05f - 0.5f;      // (b + 1/2) / 2^16 - 1/2
  float rad = sqrtf(-2.0f * __logf(u1));
  float sn, cs;
  __sincosf(6.283185307179586f * u2, &sn, &cs);   // angle in (-pi, pi)
  n0 = rad * cs;
  n1 = rad * sn;
}

// Three standard complex normals (one per parameter) for bin (i,j,k) of realisation s,
// Hermitian-consistent on the planes whose x-bin is its own mirror (i = 0, and
// i = nxp/2 for even nxp): the pair (j,k) / (-j,-k) share one draw (conjugated),
// self-mirrored bins are real with unit variance, all others have variance 1/2 per
// component (the properties FFTGrid::fillInComplexNoise gives its noise,
// src/fftgrid.cpp:997-1055, with the mirror-plane test done on the x index).  One
// Philox block (128 bits) per bin and realisation feeds the three Box-Muller pairs: three
// 26-bit radius words (the top bits of words 0-2) and three 16-bit angle words (word 3's two
// halves, and the low 6 + 6 + 4 bits of words 0-2).
__device__ __forceinline__ void device_noise3(uint64_t seed, int s, int i, int j, int k, int nyp, int nzp,
                                              int cnxp, bool nxp_even, float2 (&z)[3]) {
  bool mirror_plane = (i == 0) || (nxp_even && i == cnxp - 1);
  int jj = j, kk = k;
  bool conj = false, self = false;
  if (mirror_plane) {
    int jc = j == 0 ? 0 : nyp - j;
    int kc = k == 0 ? 0 : nzp - k;
    long long a = (long long)j + (long long)nyp * k, b = (long long)jc + (long long)nyp * kc;
    if (a == b) self = true;
    else if (b < a) { jj = jc; kk = kc; conj = true; }
  }
  uint64_t bin = ((uint64_t)kk * nyp + jj) * cnxp + i;
  uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const uint4 r = philox4x32_7(make_uint4((uint32_t)bin, (uint32_t)(bin >> 32), (uint32_t)s, 0u), key);
  const uint32_t b2 = (r.x & 63u) | ((r.y & 63u) << 6) | ((r.z & 15u) << 12);
  float n[6];
  box_muller(r.x >> 6, r.w & 0xFFFFu, n[0], n[1]);
  box_muller(r.y >> 6, r.w >> 16, n[2], n[3]);
  box_muller(r.z >> 6, b2, n[4], n[5]);
  const float h = self ? 1.0f : 0.70710678118654752f;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    z[c] = make_float2(h * n[2 * c], self ? 0.f : h * n[2 * c + 1]);
    if (conj) z[c].y = -z[c].y;
  }
}

// ------------------------------------------------------------------ per-bin algebra, eigen form

// mu_post, S_post (order 00 11 22 01 02 12) and the residual (in d) of NB bins of one z
// position from that position's row e (float4 groups at stride nzp), laid out as EigLayout:
// the angles' rows are streamed one at a time and every row load serves all NB bins.
template <int NTH, int NB>
__device__ __forceinline__ void bin_posterior_eig(const ZParams& P, const float4* __restrict__ e,
                                                  const float (&lam)[NB], const float (&rho)[NB],
                                                  const float2 (&mu)[NB][3], float2 (&d)[NB][NTH],
                                                  float2 (&mu_post)[NB][3], float2 (&sp)[NB][6]) {
  constexpr int VP = pad4(2 * NTH), OKW = 0, OL = VP, OR = OL + pad4(NTH), RS = VP + 16;
  const int st = P.nzp;
  float kw[VP];
  ldrow(kw, e + (OKW / 4) * st, st);
  float Lm[pad4(NTH)];
  ldrow(Lm, e + (OL / 4) * st, st);
  // y = d - K mu, K = diag(kw) A
  float2 y[NB][NTH];
#pragma unroll
  for (int b = 0; b < NB; b++)
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      float2 am = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < 3; a++)
        am = make_float2(am.x + P.A[l][a] * mu[b][a].x, am.y + P.A[l][a] * mu[b][a].y);
      y[b][l] = csub(d[b][l], cmul(make_float2(kw[2 * l], kw[2 * l + 1]), am));
    }
  float2 mp[NB][3];
  float s00[NB], s11[NB], s22[NB];
  float2 s01[NB], s02[NB], s12[NB];
#pragma unroll
  for (int b = 0; b < NB; b++) {
#pragma unroll
    for (int a = 0; a < 3; a++) mp[b][a] = mu[b][a];
    s00[b] = rho[b] * P.pv[0];
    s11[b] = rho[b] * P.pv[1];
    s22[b] = rho[b] * P.pv[2];
    s01[b] = make_float2(rho[b] * P.pv[3], 0.f);
    s02[b] = make_float2(rho[b] * P.pv[4], 0.f);
    s12[b] = make_float2(rho[b] * P.pv[5], 0.f);
  }
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    // r_l = (V y)_l, s_l = r_l lam / (lam Lam_l + 1), w_l = lam^2 / (lam Lam_l + 1)
    float V[VP];
    ldrow(V, e + ((OR + l * RS) / 4) * st, st);
    float QH[16];
    ldrow(QH, e + ((OR + l * RS + VP) / 4) * st, st);
    const float* h = QH + 6;
#pragma unroll
    for (int b = 0; b < NB; b++) {
      float2 r = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < NTH; m++) r = cadd(r, cmul(make_float2(V[2 * m], V[2 * m + 1]), y[b][m]));
      const float inv = __frcp_rn(fmaf(lam[b], Lm[l], 1.0f));
      const float f = lam[b] * inv;
      const float2 sl = make_float2(r.x * f, r.y * f);
      const float wl = lam[b] * f;
      // mu_post += conj(Q_l.) s_l;  S_post -= w_l H_l, H_l = (|Q_l0|^2, |Q_l1|^2, |Q_l2|^2,
      // conj(Q_l0) Q_l1, conj(Q_l0) Q_l2, conj(Q_l1) Q_l2)
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float qr = QH[2 * a], qi = QH[2 * a + 1];
        mp[b][a].x += qr * sl.x + qi * sl.y;
        mp[b][a].y += qr * sl.y - qi * sl.x;
      }
      s00[b] -= wl * h[0];
      s11[b] -= wl * h[1];
      s22[b] -= wl * h[2];
      s01[b] = make_float2(s01[b].x - wl * h[3], s01[b].y - wl * h[4]);
      s02[b] = make_float2(s02[b].x - wl * h[5], s02[b].y - wl * h[6]);
      s12[b] = make_float2(s12[b].x - wl * h[7], s12[b].y - wl * h[8]);
    }
  }
#pragma unroll
  for (int b = 0; b < NB; b++) {
#pragma unroll
    for (int a = 0; a < 3; a++) mu_post[b][a] = mp[b][a];
    sp[b][0] = make_float2(s00[b], 0.f);
    sp[b][1] = make_float2(s11[b], 0.f);
    sp[b][2] = make_float2(s22[b], 0.f);
    sp[b][3] = s01[b];
    sp[b][4] = s02[b];
    sp[b][5] = s12[b];
    // residual d - K mu_post = y - K (mu_post - mu) (the data spectrum itself where the row
    // is zero: kz not inverted)
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      float2 am = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < 3; a++)
        am = make_float2(am.x + P.A[l][a] * (mp[b][a].x - mu[b][a].x), am.y + P.A[l][a] * (mp[b][a].y - mu[b][a].y));
      d[b][l] = csub(y[b][l], cmul(make_float2(kw[2 * l], kw[2 * l + 1]), am));
    }
  }
}

// ------------------------------------------------------------------ the kernel

// Shared-memory layout of one pencil tile (W consecutive x-bins at one y, all nzp kz):
//   tw  [nzp]             z twiddles
//   R   [nzp][G][W]       G = max(nth + 3, 9) slots per bin: inputs data 0..nth-1 and
//                         mean nth..nth+2; after the per-bin step outputs S_post 0..5 and
//                         mu_post 6..8 (each bin's slots are owned by the thread of that bin)
//   SC  [GT * W * nzp]    transform scratch: the z transforms run GT slots per call
//   S3  [nzp][3 SB][W]    the output spectra of SB realisations, transformed together
// Element (slot g, kz k, x-offset w) of R is R[(k * G + g) * W + w].  3 SB <= GT.


// REFINE instantiates the FP64 re-factorisation of flagged bins; the FP32-only kernel is
// a separate instantiation so that its register allocation does not carry the call.
template <int NTH, bool REFINE>
__global__ void __launch_bounds__(512) k_zpass(const __grid_constant__ ZParams P) {
  extern __shared__ float2 sm[];
  const int nzp = P.nzp, W = P.W, lw = P.logW;
  const int TS = W * nzp;
  constexpr int G = NTH + 3 > 9 ? NTH + 3 : 9;
  constexpr int GIN = NTH + 3;
  const int GT = P.GT, SB = P.SB;
  float2* tw = sm;
  float2* R = tw + nzp;
  float2* SC = R + G * TS;
  float2* S3 = SC + GT * TS;
  __shared__ unsigned long long cnt[4];
  const int T = blockDim.x, tid = threadIdx.x;
  const int it = blockIdx.x % P.nIT;
  const int j = blockIdx.x / P.nIT;
  const int i0 = it * W;
  const int nw = min(W, P.cnxp - i0);
  const size_t kstride = (size_t)P.nyp * P.cnxp;
  const size_t base = (size_t)j * P.cnxp + i0;

  if (tid < 4) cnt[tid] = 0;
  for (int t = tid; t < nzp; t += T) tw[t] = P.twz[t];
  // ---- load inputs: slot g <- data[g] (g < NTH) or mean[g - NTH]; every copy is issued
  //      before the first is waited for (cp.async), x-bins beyond the grid are zero-filled
  {
    const uint32_t rb = smem_addr(R);
    for (int e = tid; e < TS; e += T) {
      const int w = e & (W - 1), k = e >> lw;
      const bool ok = w < nw;
      const size_t go = base + (ok ? (size_t)k * kstride + w : 0);   // nothing is read when !ok
      const uint32_t sa = rb + 8u * (uint32_t)(k * G * W + w);
#pragma unroll
      for (int g = 0; g < GIN; g++)
        cp_async8_zfill(sa + 8u * (uint32_t)(g * W), (g < NTH ? P.data[g] : P.mean[g - NTH]) + go, ok);
    }
    cp_async_commit();
    cp_async_wait_0();
  }
  __syncthreads();
  // forward z transforms, GT slots per call
#pragma unroll 1
  for (int g0 = 0; g0 < GIN; g0 += GT) {
    int ng = min(GT, GIN - g0);
    fft_lines<true, -1>(R + g0 * W, SC, ng * W, 1, G * W, P.zp, tw);
  }

  // A NaN or Inf anywhere in a data or prior-mean grid reaches every bin through the three
  // transforms, so one bin per tile tells whether the inputs were finite.
  if (tid == 0 && P.counters) {
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < GIN; g++) s += fabsf(R[g * W].x) + fabsf(R[g * W].y);
    if (!isfinite(s)) atomicAdd(P.counters + 4, 1ull);
  }
  // ---- per-bin posterior (src/avoinversion.cpp:1016-1082)
  unsigned long long n_inv = 0, n_fail = 0, n_zero_bins = 0, n_fp64 = 0;
  for (int b = tid; b < TS; b += T) {
    int k = b >> lw, w = b & (W - 1);
    if (w >= nw) continue;
    int i = i0 + w;
    size_t gidx = base + (size_t)k * kstride + w;
    float2* slot = R + k * G * W + w;   // slot g at slot[g * W]
    float S[6], lam, rho = 0.f;
    if (P.separable) {
      float2 cx = __ldg(P.cxy + (size_t)j * P.cnxp + i);
      float2 c_t = __ldg(P.ct + k);
      rho = fabsf(cx.x * c_t.x - cx.y * c_t.y);
#pragma unroll
      for (int q = 0; q < 6; q++) S[q] = P.pv[q] * rho;
      lam = fabsf(cx.x);
    } else {
      // getNextParameterCovariance: |Re/pv| pv (no division when pv == 0); a base prior's
      // pairs share |Re/pv| of the one spectrum transformed (pv[0] != 0)
      if (P.base_prior) {
        const float r0 = fabsf(P.cov[0][gidx].x / P.pv[0]);
#pragma unroll
        for (int q = 0; q < 6; q++) S[q] = r0 * P.pv[q];
      } else {
#pragma unroll
        for (int q = 0; q < 6; q++) {
          float re = P.cov[q][gidx].x;
          float pv = P.pv[q];
          if (pv != 0.f) re = re / pv;
          S[q] = fabsf(re) * pv;
        }
      }
      lam = fabsf(P.errspec[gidx].x);
    }
    float2 mu[3], d[NTH];
#pragma unroll
    for (int a = 0; a < 3; a++) mu[a] = slot[(NTH + a) * W];
#pragma unroll
    for (int l = 0; l < NTH; l++) d[l] = slot[l * W];
    BinOut o;
    bool inv = P.kz.inv[k] != 0;
    bool ok = false;
    if (!REFINE && P.eig) {
      // separable prior with a real temporal spectrum: the eigen form of the per-bin step
      // (bin_posterior_eig, tables in natural kz order), which never needs a fallback (the
      // host bounds the lateral factor against the reference's pivot test before choosing it)
      const float lam1[1] = {lam}, rho1[1] = {rho};
      float2 mu1[1][3], d1[1][NTH], mp1[1][3], sp1[1][6];
#pragma unroll
      for (int a = 0; a < 3; a++) mu1[0][a] = mu[a];
#pragma unroll
      for (int l = 0; l < NTH; l++) d1[0][l] = d[l];
      bin_posterior_eig<NTH, 1>(P, P.eig + k, lam1, rho1, mu1, d1, mp1, sp1);
#pragma unroll
      for (int a = 0; a < 3; a++) o.mu[a] = mp1[0][a];
#pragma unroll
      for (int q = 0; q < 6; q++) o.sp[q] = sp1[0][q];
#pragma unroll
      for (int l = 0; l < NTH; l++) d[l] = d1[0][l];
      if (inv) n_inv++;
      ok = true;
    } else if (inv) {
      n_inv++;
      ok = P.septab ? bin_posterior<NTH, true>(P, k, S, lam, rho, mu, d, o)
                    : bin_posterior<NTH, false>(P, k, S, lam, rho, mu, d, o);
      if constexpr (REFINE) {
        if (ok) {
          float ratio = 1.f;
#pragma unroll
          for (int a = 0; a < 3; a++)
            if (S[a] > 0.f) ratio = fminf(ratio, o.sp[a].x / S[a]);
          if (o.cond > P.fp64_threshold || ratio * P.fp64_threshold < 1.f) {
            // the data are still in their slots: restart from them
            float2 d64[NTH];
#pragma unroll
            for (int l = 0; l < NTH; l++) d64[l] = slot[l * W];
            if (bin_posterior_fp64<NTH>(P, k, S, lam, mu, d64, o)) {
              n_fp64++;
#pragma unroll
              for (int l = 0; l < NTH; l++) d[l] = d64[l];
            }
          }
        }
      }
      if (!ok) n_fail++;
    }
    if (!ok) {
#pragma unroll
      for (int a = 0; a < 3; a++) o.mu[a] = mu[a];
#pragma unroll
      for (int q = 0; q < 6; q++) o.sp[q] = make_float2(S[q], 0.f);
    }
    if (P.keep_resid) {
#pragma unroll
      for (int l = 0; l < NTH; l++) P.data[l][gidx] = d[l];
    }
    // Factor S_post once for all realisations (lib_matrCholCpx(3), simulate :1425-1443).
    // Slots 0..5 then hold L (diagonal real, slot 0 imaginary part set to -1 as the mark)
    // or, where the factorisation fails, S_post itself; the covariance output is rebuilt
    // as L L^H before its inverse transform.
    float2 C[3][3];
    C[0][0] = o.sp[0]; C[1][1] = o.sp[1]; C[2][2] = o.sp[2];
    C[0][1] = o.sp[3]; C[0][2] = o.sp[4]; C[1][2] = o.sp[5];
    C[1][0] = make_float2(o.sp[3].x, -o.sp[3].y);
    C[2][0] = make_float2(o.sp[4].x, -o.sp[4].y);
    C[2][1] = make_float2(o.sp[5].x, -o.sp[5].y);
    if (P.nsim > 0 && chol_ref<3>(C)) {
      slot[0] = make_float2(C[0][0].x, -1.f);
      slot[W] = make_float2(C[1][1].x, 0.f);
      slot[2 * W] = make_float2(C[2][2].x, 0.f);
      slot[3 * W] = C[1][0];
      slot[4 * W] = C[2][0];
      slot[5 * W] = C[2][1];
    } else {
      if (P.nsim > 0) n_zero_bins++;
#pragma unroll
      for (int q = 0; q < 6; q++) slot[q * W] = o.sp[q];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) slot[(6 + a) * W] = o.mu[a];
  }
  __syncthreads();

  // ---- realisations (src/avoinversion.cpp:1401-1511), mean added in the spectral domain;
  //      SB realisations per batch share one transform call
#pragma unroll 1
  for (int s0 = 0; s0 < P.nsim; s0 += SB) {
    const int nb = min(SB, P.nsim - s0);
    const int SG = 3 * nb;  // slots of this batch
    for (int b = tid; b < TS; b += T) {
      int k = b >> lw, w = b & (W - 1);
      float2* o3 = S3 + k * SG * W + w;
      if (w >= nw) {
        for (int q = 0; q < SG; q++) o3[q * W] = make_float2(0.f, 0.f);
        continue;
      }
      int i = i0 + w;
      size_t gidx = base + (size_t)k * kstride + w;
      const float2* slot = R + k * G * W + w;
      const float2 l0 = slot[0];
      const float2 m0 = slot[6 * W], m1 = slot[7 * W], m2 = slot[8 * W];
#pragma unroll 1
      for (int sb = 0; sb < nb; sb++) {
        const int s = s0 + sb;
        float2 sd[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (l0.y == -1.f) {
          float2 z[3];
          if (P.host_noise) {
#pragma unroll
            for (int c = 0; c < 3; c++) z[c] = P.noise[3 * s + c][gidx];
          } else {
            device_noise3(P.seed, s, i, j, k, P.nyp, nzp, P.cnxp, P.nxp_even, z);
          }
          const float2 l1 = slot[W], l2 = slot[2 * W], l10 = slot[3 * W], l20 = slot[4 * W], l21 = slot[5 * W];
          sd[0] = make_float2(l0.x * z[0].x, l0.x * z[0].y);
          sd[1] = cadd(cmul(l10, z[0]), make_float2(l1.x * z[1].x, l1.x * z[1].y));
          sd[2] = cadd(cadd(cmul(l20, z[0]), cmul(l21, z[1])), make_float2(l2.x * z[2].x, l2.x * z[2].y));
        }
        o3[(3 * sb + 0) * W] = cadd(m0, sd[0]);
        o3[(3 * sb + 1) * W] = cadd(m1, sd[1]);
        o3[(3 * sb + 2) * W] = cadd(m2, sd[2]);
      }
    }
    __syncthreads();
    const float2* res = S3;
    fft_lines<true, 1>(S3, SC, SG * W, 1, SG * W, P.zp, tw);
    for (int e = tid; e < TS; e += T) {
      const int w = e & (W - 1), k = e >> lw;
      if (w >= nw) continue;
      const size_t go = base + (size_t)k * kstride + w;
      const float2* r = res + k * SG * W + w;
#pragma unroll
      for (int q = 0; q < 6; q++)
        if (q < SG) P.sim[3 * s0 + q][go] = r[q * W];
    }
    __syncthreads();
  }
  // ---- rebuild S_post = L L^H where slots 0..5 hold the factor
  if (P.nsim > 0) {
    for (int b = tid; b < TS; b += T) {
      int k = b >> lw, w = b & (W - 1);
      float2* slot = R + k * G * W + w;
      const float2 l0 = slot[0];
      if (l0.y != -1.f) continue;
      const float2 l1 = slot[W], l2 = slot[2 * W], l10 = slot[3 * W], l20 = slot[4 * W], l21 = slot[5 * W];
      // S_ab = sum_c L_ac conj(L_bc)
      slot[0] = make_float2(l0.x * l0.x, 0.f);
      slot[W] = make_float2(l10.x * l10.x + l10.y * l10.y + l1.x * l1.x, 0.f);
      slot[2 * W] = make_float2(l20.x * l20.x + l20.y * l20.y + l21.x * l21.x + l21.y * l21.y + l2.x * l2.x, 0.f);
      slot[3 * W] = make_float2(l0.x * l10.x, -l0.x * l10.y);
      slot[4 * W] = make_float2(l0.x * l20.x, -l0.x * l20.y);
      slot[5 * W] = make_float2(l10.x * l20.x + l10.y * l20.y + l1.x * l21.x,
                                l10.y * l20.x - l10.x * l20.y - l1.x * l21.y);
    }
    __syncthreads();
  }

  // ---- inverse z transform of posterior covariance (slots 0..5, unless it stays spectral)
  //      and mean (6..8)
  const int gs0 = P.cov_spectral ? 6 : 0;
#pragma unroll 1
  for (int g0 = gs0; g0 < 9; g0 += GT)
    fft_lines<true, 1>(R + g0 * W, SC, min(GT, 9 - g0) * W, 1, G * W, P.zp, tw);
  for (int e = tid; e < TS; e += T) {
    const int w = e & (W - 1), k = e >> lw;
    if (w >= nw) continue;
    const size_t go = base + (size_t)k * kstride + w;
    const int so = k * G * W + w;
#pragma unroll
    for (int g = 0; g < 9; g++) {
      (g < 6 ? P.cov[g] : P.mean[g - 6])[go] = R[so + g * W];
    }
  }

  // counters
  unsigned long long n_zero = n_zero_bins * (unsigned long long)P.nsim;
  for (int off = 16; off > 0; off >>= 1) {
    n_inv += __shfl_down_sync(0xffffffffu, n_inv, off);
    n_fail += __shfl_down_sync(0xffffffffu, n_fail, off);
    n_zero += __shfl_down_sync(0xffffffffu, n_zero, off);
    n_fp64 += __shfl_down_sync(0xffffffffu, n_fp64, off);
  }
  if ((tid & 31) == 0) {
    atomicAdd(&cnt[0], n_inv);
    atomicAdd(&cnt[1], n_fail);
    atomicAdd(&cnt[2], n_zero);
    atomicAdd(&cnt[3], n_fp64);
  }
  __syncthreads();
  if (tid == 0 && P.counters) {
    atomicAdd(P.counters + 0, cnt[0]);
    atomicAdd(P.counters + 1, cnt[1]);
    atomicAdd(P.counters + 2, cnt[2]);
    atomicAdd(P.counters + 3, cnt[3]);
  }
}

// ------------------------------------------------------------------ launch templates

template <int NTH, bool REFINE>
inline cudaError_t launch_zpass_r(const ZParams& zp, int threads, cudaStream_t st) {
  size_t smem = zpass_smem_bytes(zp.W, zp.nzp, zp.nth, zp.GT, zp.SB);
  cudaError_t e = cudaFuncSetAttribute(k_zpass<NTH, REFINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)(zp.nIT * zp.nyp));
  k_zpass<NTH, REFINE><<<grid, threads, smem, st>>>(zp);
  return cudaGetLastError();
}

template <int NTH>
inline cudaError_t launch_zpass_t(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.fp64_threshold > 0.f ? launch_zpass_r<NTH, true>(zp, threads, st)
                                 : launch_zpass_r<NTH, false>(zp, threads, st);
}

// the general kernel's launchers by angle count (zpass_n12.cu, zpass_n34.cu, zpass_n56.cu,
// zpass_n78.cu): one translation unit per pair so that they compile side by side
cudaError_t launch_zpass_n12(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_zpass_n34(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_zpass_n56(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_zpass_n78(const ZParams& zp, int threads, cudaStream_t st);

}  // namespace crava

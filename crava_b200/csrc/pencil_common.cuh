// Device helpers of the pencil pass (pencil.cuh, pencil_bin.cuh): the counter-based noise of
// product-mode realisations and the reference-semantics Cholesky factorisation of small
// Hermitian matrices.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_pair.cuh"
#include "kernels.cuh"

namespace crava {

// ------------------------------------------------------------------ noise (product mode)

// Philox-4x32 (Salmon, Moraes, Dror, Shaw, SC'11) with 7 rounds, which the authors
// report passes TestU01 BigCrush.
__device__ __forceinline__ uint4 philox4x32_7(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 7; r++) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k.x, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k.y, (uint32_t)p0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

// Three standard complex normals (one per parameter) for each of the bins (i,j,k) and (i+1,j,k) of
// realisation s, Hermitian-consistent on the planes whose x-bin is its own mirror (i = 0, and
// i = nxp/2 for even nxp): the pair (j,k) / (-j,-k) share one draw (conjugated),
// self-mirrored bins are real with unit variance, all others have variance 1/2 per
// component (the properties FFTGrid::fillInComplexNoise gives its noise,
// src/fftgrid.cpp:997-1055, with the mirror-plane test done on the x index).  One
// Philox block (128 bits) per bin and realisation feeds the three Box-Muller pairs: three
// 26-bit radius words a (the top bits of words 0-2) and three 16-bit angle words b (word 3's two
// halves, and the low 6 + 6 + 4 bits of words 0-2).  Box-Muller takes u1 = (a + 1/2) / 2^26
// (the largest |normal| is sqrt(2 ln 2^27) = 6.1) and the angle 2 pi ((b + 1/2) / 2^16 - 1/2), with the
// hardware approximations of log, sine and cosine: their absolute errors (about 2^-21 on
// these ranges) are far below what the normals' statistics can show.  The two bins' arithmetic is
// packed, with the operations and roundings of device_noise3 (zpass.cuh), so that a bin's draw does not
// depend on the kernel that makes it; b / 2^16 comes from the mantissa bits of [1, 2) without a
// conversion.
__device__ __forceinline__ void pair_noise(const ZParams& P, int s, int i, int j, int k, C2 (&z)[3]) {
  const int last = P.cnxp - 1;
  uint64_t bin[2];
  bin[0] = ((uint64_t)(uint32_t)k * (uint32_t)P.nyp + (uint32_t)j) * (uint32_t)P.cnxp + (uint64_t)(int64_t)i;
  bin[1] = bin[0] + 1;
  const bool edge = i <= 0 || i + 1 >= last;
  bool self[2] = {false, false}, conj[2] = {false, false};
  if (edge) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (i + u != 0 && !(P.nxp_even && i + u == last)) continue;
      const int jc = j == 0 ? 0 : P.nyp - j, kc = k == 0 ? 0 : P.nzp - k;
      const long long a = (long long)j + (long long)P.nyp * k, b = (long long)jc + (long long)P.nyp * kc;
      if (a == b) self[u] = true;
      else if (b < a) {
        conj[u] = true;
        bin[u] = ((uint64_t)kc * P.nyp + jc) * P.cnxp + (i + u);
      }
    }
  }
  constexpr float kH = 0.70710678118654752f;
  const float2 h = make_float2(self[0] ? 1.0f : kH, self[1] ? 1.0f : kH);
  const uint2 key = make_uint2((uint32_t)P.seed, (uint32_t)(P.seed >> 32));
  uint4 r[2];
#pragma unroll
  for (int u = 0; u < 2; u++)
    r[u] = philox4x32_7(make_uint4((uint32_t)bin[u], (uint32_t)(bin[u] >> 32), (uint32_t)s, 0u), key);
  uint32_t b[3][2];
#pragma unroll
  for (int u = 0; u < 2; u++) {   // 1 + b / 2^16 as float bits
    b[0][u] = 0x3F800000u | ((r[u].w << 7) & 0x7FFF80u);
    b[1][u] = 0x3F800000u | ((r[u].w >> 9) & 0x7FFF80u);
    b[2][u] = 0x3F800000u | ((r[u].x & 63u) << 7) | ((r[u].y & 63u) << 13) | ((r[u].z & 15u) << 19);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const uint32_t a0 = (c == 0 ? r[0].x : c == 1 ? r[0].y : r[0].z) >> 6;
    const uint32_t a1 = (c == 0 ? r[1].x : c == 1 ? r[1].y : r[1].z) >> 6;
    const float2 u1 = f2_mul(f2_add(make_float2((float)a0, (float)a1), f2_dup(0.5f)), f2_dup(1.4901161193847656e-08f));
    const float2 t = f2_mul(make_float2(__logf(u1.x), __logf(u1.y)), f2_dup(-2.0f));
    const float2 rad = make_float2(sqrtf(t.x), sqrtf(t.y));
    // (1 + b / 2^16) - (3/2 - 2^-17), exact
    const float2 u2 = f2_add(make_float2(__uint_as_float(b[c][0]), __uint_as_float(b[c][1])), f2_dup(-1.49999237060546875f));
    const float2 ang = f2_mul(u2, f2_dup(6.283185307179586f));   // in (-pi, pi)
    float2 sn, cs;
    __sincosf(ang.x, &sn.x, &cs.x);
    __sincosf(ang.y, &sn.y, &cs.y);
    z[c] = {f2_mul(f2_mul(rad, cs), h), f2_mul(f2_mul(rad, sn), h)};
  }
  if (edge) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (self[0]) z[c].i.x = 0.f;
      else if (conj[0]) z[c].i.x = -z[c].i.x;
      if (self[1]) z[c].i.y = 0.f;
      else if (conj[1]) z[c].i.y = -z[c].i.y;
    }
  }
}

// ------------------------------------------------------------------ per-bin algebra

// lib_matrCholCpx (libs/lib/lib_matr.c:78-168) on the lower triangle of a Hermitian
// n x n matrix a[][]: the reference scales by a00, rejects a00 <= 0, a scaled diagonal
// <= 1e-20 before its update or an updated pivot <= 1e-20, factors and rescales by
// sqrt(a00).  Here the factor is computed unscaled with the two pivot tests applied as
// a_ii > 1e-20 a00 (the same comparisons up to rounding), and each pivot's reciprocal
// comes from one reciprocal square root.  No division.  The diagonal entry holds
// (L_ii, 1 / L_ii): its imaginary part, zero for a Hermitian factor, carries the reciprocal.
template <int N>
__device__ __forceinline__ bool chol_ref(float2 (&a)[N][N]) {
  const float f = a[0][0].x;
  if (!(f > 0.f)) return false;
  const float tol = 1e-20f * f;
#pragma unroll
  for (int i = 0; i < N; i++) {
    if (!(a[i][i].x > tol)) return false;
#pragma unroll
    for (int j = 0; j < i; j++) {
      float2 s = a[i][j];
#pragma unroll
      for (int k = 0; k < j; k++) {  // - L_ik conj(L_jk)
        s.x -= a[i][k].x * a[j][k].x + a[i][k].y * a[j][k].y;
        s.y -= -(a[i][k].x * a[j][k].y) + a[i][k].y * a[j][k].x;
      }
      a[i][j] = make_float2(s.x * a[j][j].y, s.y * a[j][j].y);
    }
    float r = a[i][i].x;
#pragma unroll
    for (int k = 0; k < i; k++) r -= a[i][k].x * a[i][k].x + a[i][k].y * a[i][k].y;
    if (!(r > tol)) return false;
    const float rs = rsqrtf(r);
    a[i][i] = make_float2(r * rs, rs);
  }
  return true;
}

// ------------------------------------------------------------------ eigen tables

constexpr int pad4(int x) { return (x + 3) / 4 * 4; }

// Section of N floats (N % 4 == 0) of the row of position p: group g at e[g * stride].
template <int N>
__device__ __forceinline__ void ldrow(float (&out)[N], const float4* __restrict__ e, int stride) {
#pragma unroll
  for (int g = 0; g < N / 4; g++) {
    const float4 v = __ldg(e + g * stride);
    out[4 * g] = v.x;
    out[4 * g + 1] = v.y;
    out[4 * g + 2] = v.z;
    out[4 * g + 3] = v.w;
  }
}

}  // namespace crava

// The per-bin posterior by a Cholesky factorisation of the data covariance (sm_100a): the form the
// pencil pass (pencil.cuh) takes where its eigen form does not apply -- prior grids, a temporal
// correlation that is not symmetric, and the FP64 re-factorisation of ill-conditioned bins.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_core.cuh"
#include "kernels.cuh"
#include "pencil_common.cuh"

namespace crava {

struct BinOut {
  float2 mu[3];
  float2 sp[6];
  float cond;   // (max / min Cholesky pivot)^2 of Sd, an estimate of its condition number
};

// Posterior of one bin.  Follows src/avoinversion.cpp:1036-1061 with
//   Sd = K S K^H + Se, K = diag(kw) A, S real symmetric (so K S K^H = (kw kw^H) o (A S A^T)),
//   L L^H = Sd (reference Cholesky), Y = L^{-1} K S,
//   S_post = S - Y^H Y, mu_post = mu + Y^H L^{-1} (d - K mu), res = d - K mu_post,
// which is the reference's  KS <- Sd^{-1} KS; S - KS_old^H KS;  mu + KS^H (d - K mu)
// regrouped through the Cholesky factor.
// SEP: separable prior.  Then S = rho P0, so K S K^H = rho (kw kw^H) o G0 and K S = rho
// diag(kw) AP with G0 = A P0 A^T and AP = A P0 job constants, and the error part of Sd is
// lam M2 with M2 = ec o (e1 e1^H + e2 e2^H) read per kz from the job's table (lower
// triangle, row by row), in place of the per-bin products.
template <int NTH, bool SEP>
__device__ __forceinline__ bool bin_posterior(const ZParams& P, int k, const float (&S)[6], float lam, float rho,
                                              const float2 (&mu)[3], float2 (&d)[NTH], BinOut& o) {
  constexpr int TRI = NTH * (NTH + 1) / 2;
  float2 kw[NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) kw[l] = __ldg(P.kz.kw + k * NTH + l);
  float2 Sd[NTH][NTH];
  float2 Y[NTH][3];  // K S, then L^{-1} K S
  if constexpr (SEP) {
    const float2* m2 = P.septab + (size_t)k * TRI;
#pragma unroll
    for (int l = 0; l < NTH; l++) {
#pragma unroll
      for (int m = 0; m <= l; m++) {
        const float2 b = __ldg(m2 + l * (l + 1) / 2 + m);
        const float g = rho * P.G0[l][m];
        // rho G0_lm kw_l conj(kw_m) + lam M2_lm
        Sd[l][m] = make_float2(g * (kw[l].x * kw[m].x + kw[l].y * kw[m].y) + lam * b.x,
                               g * (kw[l].y * kw[m].x - kw[l].x * kw[m].y) + lam * b.y);
      }
      Sd[l][l] = make_float2(Sd[l][l].x + __ldg(P.kz.ed + k * NTH + l), 0.f);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const float a = rho * P.AP[l][j];
        Y[l][j] = make_float2(kw[l].x * a, kw[l].y * a);
      }
    }
  } else {
    float2 e1[NTH], e2[NTH];
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      e1[l] = __ldg(P.kz.e1 + k * NTH + l);
      e2[l] = __ldg(P.kz.e2 + k * NTH + l);
    }
    // AS = A S (NTH x 3), G = A S A^T
    float AS[NTH][3];
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      AS[l][0] = P.A[l][0] * S[0] + P.A[l][1] * S[3] + P.A[l][2] * S[4];
      AS[l][1] = P.A[l][0] * S[3] + P.A[l][1] * S[1] + P.A[l][2] * S[5];
      AS[l][2] = P.A[l][0] * S[4] + P.A[l][1] * S[5] + P.A[l][2] * S[2];
    }
#pragma unroll
    for (int l = 0; l < NTH; l++) {
#pragma unroll
      for (int m = 0; m <= l; m++) {
        float g = AS[l][0] * P.A[m][0] + AS[l][1] * P.A[m][1] + AS[l][2] * P.A[m][2];
        // kw_l conj(kw_m)
        float2 kk = make_float2(kw[l].x * kw[m].x + kw[l].y * kw[m].y, kw[l].y * kw[m].x - kw[l].x * kw[m].y);
        float c = P.ec[l][m] * lam;
        float2 ee = make_float2(e1[l].x * e1[m].x + e1[l].y * e1[m].y + e2[l].x * e2[m].x + e2[l].y * e2[m].y,
                                e1[l].y * e1[m].x - e1[l].x * e1[m].y + e2[l].y * e2[m].x - e2[l].x * e2[m].y);
        Sd[l][m] = make_float2(kk.x * g + c * ee.x, kk.y * g + c * ee.y);
        if (l == m)
          Sd[l][m] = make_float2(Sd[l][m].x + __ldg(P.kz.ed + k * NTH + l), 0.f);
      }
#pragma unroll
      for (int j = 0; j < 3; j++) Y[l][j] = make_float2(kw[l].x * AS[l][j], kw[l].y * AS[l][j]);
    }
  }
  if (!chol_ref<NTH>(Sd)) return false;
  {
    float dmax = Sd[0][0].x, rmax = Sd[0][0].y;
#pragma unroll
    for (int l = 1; l < NTH; l++) {
      dmax = fmaxf(dmax, Sd[l][l].x);
      rmax = fmaxf(rmax, Sd[l][l].y);
    }
    o.cond = (dmax * rmax) * (dmax * rmax);
  }
  // Y = L^{-1} KS (forward substitution in place)
#pragma unroll
  for (int l = 0; l < NTH; l++) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      float2 acc = Y[l][j];
#pragma unroll
      for (int m = 0; m < l; m++) acc = csub(acc, cmul(Sd[l][m], Y[m][j]));
      Y[l][j] = make_float2(acc.x * Sd[l][l].y, acc.y * Sd[l][l].y);
    }
  }
  // S_post = S - Y^H Y
  const int qa[6] = {0, 1, 2, 0, 0, 1}, qb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int q = 0; q < 6; q++) {
    float2 r = make_float2(0.f, 0.f);
#pragma unroll
    for (int l = 0; l < NTH; l++) {  // conj(Y[l][a]) Y[l][b]
      r.x += Y[l][qa[q]].x * Y[l][qb[q]].x + Y[l][qa[q]].y * Y[l][qb[q]].y;
      r.y += Y[l][qa[q]].x * Y[l][qb[q]].y - Y[l][qa[q]].y * Y[l][qb[q]].x;
    }
    o.sp[q] = make_float2(S[q] - r.x, -r.y);
  }
  // yd = L^{-1} (d - K mu)
  float2 yd[NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    float2 am = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 3; j++) am = make_float2(am.x + P.A[l][j] * mu[j].x, am.y + P.A[l][j] * mu[j].y);
    float2 acc = csub(d[l], cmul(kw[l], am));
#pragma unroll
    for (int m = 0; m < l; m++) acc = csub(acc, cmul(Sd[l][m], yd[m]));
    yd[l] = make_float2(acc.x * Sd[l][l].y, acc.y * Sd[l][l].y);
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    float2 r = mu[a];
#pragma unroll
    for (int l = 0; l < NTH; l++) {  // conj(Y[l][a]) yd[l]
      r.x += Y[l][a].x * yd[l].x + Y[l][a].y * yd[l].y;
      r.y += Y[l][a].x * yd[l].y - Y[l][a].y * yd[l].x;
    }
    o.mu[a] = r;
  }
  // residual d - K mu_post, returned in d
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    float2 am = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 3; j++) am = make_float2(am.x + P.A[l][j] * o.mu[j].x, am.y + P.A[l][j] * o.mu[j].y);
    d[l] = csub(d[l], cmul(kw[l], am));
  }
  return true;
}

// ------------------------------------------------------------------ FP64 re-factorisation

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// lib_matrCholCpx semantics (libs/lib/lib_matr.c:78-168) in double.
template <int N>
__device__ __forceinline__ bool chol_ref_d(double2 (&a)[N][N]) {
  const double TOLD = 1e-20;
  double f = a[0][0].x;
  if (!(f > 0.0)) return false;
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j <= i; j++) a[i][j] = make_double2(a[i][j].x / f, a[i][j].y / f);
#pragma unroll
  for (int i = 0; i < N; i++) {
    if (!(a[i][i].x > TOLD)) return false;
#pragma unroll
    for (int j = 0; j < i; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < j; k++) {
        s.x += a[i][k].x * a[j][k].x + a[i][k].y * a[j][k].y;
        s.y += -(a[i][k].x * a[j][k].y) + a[i][k].y * a[j][k].x;
      }
      double dd = a[j][j].x;
      a[i][j] = make_double2((a[i][j].x - s.x) / dd, (a[i][j].y - s.y) / dd);
    }
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < i; k++) r += a[i][k].x * a[i][k].x + a[i][k].y * a[i][k].y;
    r = a[i][i].x - r;
    if (!(r > TOLD)) return false;
    a[i][i] = make_double2(sqrt(r), 0.0);
  }
  double sf = sqrt(f);
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j <= i; j++) a[i][j] = make_double2(a[i][j].x * sf, a[i][j].y * sf);
  return true;
}

// The per-bin posterior of bin_posterior re-done in double for a bin the FP32 pass flagged
// as ill-conditioned, with one step of iterative refinement of the data solve
// x = Sd^{-1} (d - K mu): x0 from the factor, r = (d - K mu) - Sd x0, x = x0 + Sd^{-1} r.
// Out of line: only flagged bins call it, and only the REFINE instantiation of the pencil
// kernel carries the call.
template <int NTH>
__device__ __noinline__ bool bin_posterior_fp64(const ZParams& P, int k, const float (&Sf)[6], float lamf,
                                                const float2 (&mu)[3], float2 (&d)[NTH], BinOut& o) {
  double2 kw[NTH], e1[NTH], e2[NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    kw[l] = P.kz.kwd[k * NTH + l];
    e1[l] = P.kz.e1d[k * NTH + l];
    e2[l] = P.kz.e2d[k * NTH + l];
  }
  double S[6];
#pragma unroll
  for (int q = 0; q < 6; q++) S[q] = Sf[q];
  const double lam = lamf;
  double AS[NTH][3];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    AS[l][0] = P.Ad[l][0] * S[0] + P.Ad[l][1] * S[3] + P.Ad[l][2] * S[4];
    AS[l][1] = P.Ad[l][0] * S[3] + P.Ad[l][1] * S[1] + P.Ad[l][2] * S[5];
    AS[l][2] = P.Ad[l][0] * S[4] + P.Ad[l][1] * S[5] + P.Ad[l][2] * S[2];
  }
  double2 Sd[NTH][NTH], Sfull[NTH][NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
#pragma unroll
    for (int m = 0; m <= l; m++) {
      double g = AS[l][0] * P.Ad[m][0] + AS[l][1] * P.Ad[m][1] + AS[l][2] * P.Ad[m][2];
      double2 kk = make_double2(kw[l].x * kw[m].x + kw[l].y * kw[m].y, kw[l].y * kw[m].x - kw[l].x * kw[m].y);
      double c = P.ecd[l][m] * lam;
      double2 ee = make_double2(e1[l].x * e1[m].x + e1[l].y * e1[m].y + e2[l].x * e2[m].x + e2[l].y * e2[m].y,
                                e1[l].y * e1[m].x - e1[l].x * e1[m].y + e2[l].y * e2[m].x - e2[l].x * e2[m].y);
      Sd[l][m] = make_double2(kk.x * g + c * ee.x, kk.y * g + c * ee.y);
      if (l == m) Sd[l][m] = make_double2(Sd[l][m].x + (P.kz.edd ? P.kz.edd[k * NTH + l] : P.edd[l]), 0.0);
      Sfull[l][m] = Sd[l][m];
      Sfull[m][l] = make_double2(Sd[l][m].x, -Sd[l][m].y);
    }
  }
  if (!chol_ref_d<NTH>(Sd)) return false;
  // Y = L^{-1} K S, S_post = S - Y^H Y
  double2 Y[NTH][3];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double2 acc = make_double2(kw[l].x * AS[l][j], kw[l].y * AS[l][j]);
#pragma unroll
      for (int m = 0; m < l; m++) acc = zsub(acc, zmul(Sd[l][m], Y[m][j]));
      Y[l][j] = make_double2(acc.x / Sd[l][l].x, acc.y / Sd[l][l].x);
    }
  }
  const int qa[6] = {0, 1, 2, 0, 0, 1}, qb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int q = 0; q < 6; q++) {
    double2 r = make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      r.x += Y[l][qa[q]].x * Y[l][qb[q]].x + Y[l][qa[q]].y * Y[l][qb[q]].y;
      r.y += Y[l][qa[q]].x * Y[l][qb[q]].y - Y[l][qa[q]].y * Y[l][qb[q]].x;
    }
    o.sp[q] = make_float2((float)(S[q] - r.x), (float)(-r.y));
  }
  // b = d - K mu; x = Sd^{-1} b with one refinement step
  double2 b[NTH], x[NTH], t[NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    double2 am = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 3; j++) am = make_double2(am.x + P.Ad[l][j] * mu[j].x, am.y + P.Ad[l][j] * mu[j].y);
    b[l] = zsub(make_double2(d[l].x, d[l].y), zmul(kw[l], am));
  }
  auto solve = [&](const double2 (&rhs)[NTH], double2 (&out)[NTH]) {
#pragma unroll
    for (int l = 0; l < NTH; l++) {
      double2 acc = rhs[l];
#pragma unroll
      for (int m = 0; m < l; m++) acc = zsub(acc, zmul(Sd[l][m], t[m]));
      t[l] = make_double2(acc.x / Sd[l][l].x, acc.y / Sd[l][l].x);
    }
#pragma unroll
    for (int l = NTH - 1; l >= 0; l--) {
      double2 acc = t[l];
#pragma unroll
      for (int m = l + 1; m < NTH; m++) acc = zsub(acc, zmul(make_double2(Sd[m][l].x, -Sd[m][l].y), out[m]));
      out[l] = make_double2(acc.x / Sd[l][l].x, acc.y / Sd[l][l].x);
    }
  };
  solve(b, x);
  double2 r[NTH], dx[NTH];
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    double2 acc = b[l];
#pragma unroll
    for (int m = 0; m < NTH; m++) acc = zsub(acc, zmul(Sfull[l][m], x[m]));
    r[l] = acc;
  }
  solve(r, dx);
#pragma unroll
  for (int l = 0; l < NTH; l++) x[l] = make_double2(x[l].x + dx[l].x, x[l].y + dx[l].y);
  // mu_post = mu + (K S)^H x, residual d - K mu_post
  double2 mp[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    double2 acc = make_double2(mu[a].x, mu[a].y);
#pragma unroll
    for (int l = 0; l < NTH; l++) {  // conj(kw_l AS[l][a]) x_l
      double2 ks = make_double2(kw[l].x * AS[l][a], -kw[l].y * AS[l][a]);
      acc = make_double2(acc.x + ks.x * x[l].x - ks.y * x[l].y, acc.y + ks.x * x[l].y + ks.y * x[l].x);
    }
    mp[a] = acc;
    o.mu[a] = make_float2((float)acc.x, (float)acc.y);
  }
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    double2 am = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 3; j++) am = make_double2(am.x + P.Ad[l][j] * mp[j].x, am.y + P.Ad[l][j] * mp[j].y);
    double2 rr = zsub(make_double2(d[l].x, d[l].y), zmul(kw[l], am));
    d[l] = make_float2((float)rr.x, (float)rr.y);
  }
  return true;
}

}  // namespace crava

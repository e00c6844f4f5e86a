// The pencil pass (sm_100a).
//
// Per (x-tile, y) pencil: forward z transform of the data and prior-mean spectra, the per-bin
// posterior of AVOInversion::computePostMeanResidAndFFTCov (src/avoinversion.cpp:944-1091), the
// realisations of AVOInversion::simulate (src/avoinversion.cpp:1401-1511) and the inverse z
// transform of every output spectrum, with the spectra kept on chip between the two transforms.
//
// The per-bin algebra, eigen form.  With a separable prior whose temporal factor has a real
// spectrum (a symmetric circular correlation, as SeismicParametersHolder::computeCircCorrT builds
// it, src/seismicparametersholder.cpp:624-660), every bin of one kz has the data covariance
//     Sd = lam M_k + E_k,   M_k = |ct_k| (kw kw^H) o G0 + M2_k,   E_k = diag(ed_k) > 0,
// with lam = |Re corrXY-spectrum(i, j)| the only lateral variable, and K S = lam |ct_k|
// diag(kw) A P0.  From the Hermitian eigen-decomposition E^-1/2 M_k E^-1/2 = U diag(Lam) U^H
// (per kz, on the host, in double) and V = U^H E^-1/2, Q = |ct_k| V diag(kw) A P0:
//     mu_post = mu + lam Q^H diag(1 / (lam Lam + 1)) V (d - K mu)
//     S_post  = rho P0 - lam^2 sum_l conj(Q_la) Q_lb / (lam Lam_l + 1)
//     resid   = d - K mu_post
// which equals the reference's Sd^-1 regrouping exactly in exact arithmetic: a few small
// matrix-vector products per bin instead of a per-bin Cholesky factorisation and solves.
// Sd is positive definite for every lam >= 0 (Sd >= E_k), so the reference's Cholesky
// never falls back here; the host checks that before it chooses this form.  Elsewhere the bins
// take the Cholesky form of pencil_bin.cuh.
//
// Pairs.  Everything is done for two neighbouring x-bins at once (C2, fft_pair.cuh): the tile holds
// the bins 2 q and 2 q + 1 of a line as {re, re', im, im'}, one 16-byte word, so the transforms, the
// per-bin products and the realisations are packed FP32 instructions and their shared-memory
// accesses 16-byte ones.  Where the z stride is an even number of bins and the grids are 16-byte
// aligned (P.vec), the tiles of a row that starts on an odd bin begin one bin early, so that every
// pair is one 16-byte global access; elsewhere pairs move as two 8-byte ones.
//
// The z transforms run in place with any split of nzp into radices up to 20: stage s of the
// forward transform leaves the digits of kz reversed (position p holds kz = pencil_kz(p)), the
// per-bin step reads its tables in position order, and the inverse stages take that order back to
// natural order, the last one storing to global memory.  The stages are separate functions, one per
// radix, so that every length shares them and the kernel is instantiated by angle count alone.
//
// The diagonal of S_post is real: the pair's second bin goes into the imaginary part of the first
// one's line, which halves its share of the inverse transform (9 output spectra cost 7.5 lines) and
// of the tile; the two are told apart after the transform by S(z) = conj S(-z), each with the rounding of the
// larger (1e-7 of it: what the x transform that follows makes of a line's points in any case).
//
// What bounds it: the latency of packed chains, shared memory and barriers at 16 warps an SM (128
// registers, the tile in most of the shared memory), not HBM.  Against the scalar kernels with one
// bin a lane (5 angles, 4 realisations unless noted; ms):
//     540x540x256              6.52 -> 5.21   (25 % of the copy bandwidth)
//     768x768x320, 6 angles, 1 13.16 -> 10.18
//     270x270x256              1.60 -> 1.25   (999 -> 627 M warp instructions, 44 % of the issue slots)
//     250x250x200              2.18 -> 1.28
//     105x135x125, 16          0.61 -> 0.53
//     200x216x200, prior grids 1.35 -> 0.74, with FP64 0.82
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_pair.cuh"
#include "kernels.cuh"
#include "pencil_bin.cuh"
#include "pencil_common.cuh"

namespace crava {

// ------------------------------------------------------------------ z transforms in place
//
// Line l of nl at byte base + 16 l (+ gap from line split on), its point p ps bytes further.  A
// stage of radix R works on blocks of R sub points: v[m] at b R sub + t + sub m, t < sub.
//   forward (DIR -1): DFT over m, times w^(t k) (w = e^{-2 pi i / (R sub)}), back to sub k
//   inverse (DIR +1): times conj w^(t k), DFT over k, back to sub m
// tw: the table of e^{-2 pi i t / n}, so w = tw[tws], tws = n / (R sub).  AOS: the points come as
// {re, im, re', im'} (the way the input copies leave them).
constexpr int even_up_z(int n) { return (n + 1) & ~1; }

struct ZStage {
  uint32_t base, tw;
  int nl, ps, split, gap, items, sub, tws;
};

template <int R, int DIR>
__device__ __forceinline__ void z_twiddle(C2 (&v)[R], uint32_t tw, int step) {
#pragma unroll
  for (int k = 1; k < R; k++) {
    const float2 w = lds2(tw + 8u * (uint32_t)(step * k));
    v[k] = c2_mul(v[k], w.x, DIR < 0 ? w.y : -w.y);
  }
}

__device__ __forceinline__ uint32_t z_line(const ZStage& a, int l) {
  return a.base + 16u * (uint32_t)l + (l >= a.split ? (uint32_t)a.gap : 0u);
}

// one item of a stage: R points from byte ad on, st bytes apart; tstep: t tws, or 0
template <int R, int DIR, bool AOS>
__device__ __forceinline__ void z_load(C2 (&v)[R], uint32_t ad, uint32_t st) {
#pragma unroll
  for (int m = 0; m < R; m++) {
    if constexpr (AOS) {
      const float4 x = lds4(ad + m * st);
      v[m] = {make_float2(x.x, x.z), make_float2(x.y, x.w)};
    } else {
      v[m] = lds_c2(ad + m * st);
    }
  }
}
template <int R, int DIR, bool AOS, bool TW>
__device__ __forceinline__ void z_item(uint32_t ad, uint32_t st, uint32_t tw, int tstep) {
  C2 v[R];
  z_load<R, DIR, AOS>(v, ad, st);
  if (DIR > 0 && TW) z_twiddle<R, DIR>(v, tw, tstep);
  DftP<R, DIR>::run(v);
  if (DIR < 0 && TW) z_twiddle<R, DIR>(v, tw, tstep);
#pragma unroll
  for (int m = 0; m < R; m++) sts_c2(ad + m * st, v[m]);
}

template <int R, int DIR, bool AOS>
__device__ __noinline__ void z_stage(ZStage a) {
  const float rl = __frcp_rn((float)a.nl), rs = __frcp_rn((float)a.sub);
  const uint32_t st = (uint32_t)(a.sub * a.ps);
  for (int q = threadIdx.x; q < a.items; q += blockDim.x) {
    int l, t;
    const int j = fdivmod(q, a.nl, rl, l);
    const int b = fdivmod(j, a.sub, rs, t);
    const uint32_t ad = z_line(a, l) + (uint32_t)((b * R * a.sub + t) * a.ps);
    if (a.sub > 1) z_item<R, DIR, AOS, true>(ad, st, a.tw, t * a.tws);
    else z_item<R, DIR, AOS, false>(ad, st, a.tw, 0);
  }
}

// The last inverse stage (one block, sub = n / R): lines below split leave for global memory in
// natural order -- line l is slot l / NP, pair l % NP, and goes to out[slot] + base + k kstride at
// its two x-offsets, those in [wlo, nw) -- the others stay in place.
struct ZOut {
  uint32_t out;          // shared-memory address of the slots' grid pointers
  size_t base, kstride;
  int wlo, nw, logNP, vec;
};
// item t of line l; gs: global stride between its outputs
template <int R, bool TW>
__device__ __forceinline__ void z_last_item(const ZStage& a, const ZOut& o, int l, int t, uint32_t st, size_t gs) {
  const uint32_t ad = z_line(a, l) + (uint32_t)(t * a.ps);
  C2 v[R];
  z_load<R, 1, false>(v, ad, st);
  if (TW) z_twiddle<R, 1>(v, a.tw, t * a.tws);
  DftP<R, 1>::run(v);
  if (l >= a.split) {
#pragma unroll
    for (int m = 0; m < R; m++) sts_c2(ad + m * st, v[m]);
    return;
  }
  const int w = 2 * (l & ((1 << o.logNP) - 1));
  unsigned long long gp;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(gp) : "r"(o.out + 8u * (uint32_t)(l >> o.logNP)));
  float2* g = reinterpret_cast<float2*>(gp) + o.base + (size_t)t * o.kstride + w;
  const bool in0 = w >= o.wlo && w < o.nw, in1 = w + 1 < o.nw;
  if (o.vec && in0 && in1) {
#pragma unroll
    for (int m = 0; m < R; m++, g += gs)
      *reinterpret_cast<float4*>(g) = make_float4(v[m].r.x, v[m].i.x, v[m].r.y, v[m].i.y);
  } else {
#pragma unroll
    for (int m = 0; m < R; m++, g += gs) {
      if (in0) g[0] = make_float2(v[m].r.x, v[m].i.x);
      if (in1) g[1] = make_float2(v[m].r.y, v[m].i.y);
    }
  }
}
template <int R>
__device__ __noinline__ void z_last(ZStage a, ZOut o) {
  const float rl = __frcp_rn((float)a.nl);
  const uint32_t st = (uint32_t)(a.sub * a.ps);
  const size_t gs = (size_t)a.sub * o.kstride;
  for (int q = threadIdx.x; q < a.items; q += blockDim.x) {
    int l;
    const int t = fdivmod(q, a.nl, rl, l);
    if (a.sub > 1) z_last_item<R, true>(a, o, l, t, st, gs);
    else z_last_item<R, false>(a, o, l, t, st, gs);
  }
}

#define CRAVA_Z_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16) X(18) X(20)

template <int DIR, bool AOS>
__device__ __forceinline__ void z_stage_any(int R, const ZStage& a) {
  switch (R) {
#define CRAVA_CASE(RR) \
  case RR: z_stage<RR, DIR, AOS>(a); break;
    CRAVA_Z_RADICES(CRAVA_CASE)
#undef CRAVA_CASE
  }
}
__device__ __forceinline__ void z_last_any(int R, const ZStage& a, const ZOut& o) {
  switch (R) {
#define CRAVA_CASE(RR) \
  case RR: z_last<RR>(a, o); break;
    CRAVA_Z_RADICES(CRAVA_CASE)
#undef CRAVA_CASE
  }
}

// All stages; the caller synchronises before, every stage ends with a barrier.  R0 = 0: any plan, one
// call per stage; R0 x R1: that split inlined, its strides constants (256 points, 5 angles, 4
// realisations: about 300 of 2570 instructions a bin are the calls' own).
static __device__ __noinline__ void z_forward_any(const ZPlan& z, ZStage a) {
  int len = z.n;
  for (int s = 0; s < z.ns; s++) {
    const int R = z.radix[s];
    a.sub = len / R;
    a.tws = z.n / len;
    a.items = a.nl * (z.n / R);
    if (s == 0) z_stage_any<-1, true>(R, a);
    else z_stage_any<-1, false>(R, a);
    len = a.sub;
    __syncthreads();
  }
}
// the last stage stores the lines below split through o
static __device__ __noinline__ void z_inverse_any(const ZPlan& z, ZStage a, const ZOut& o) {
  int len = 1;
  for (int s = z.ns - 1; s >= 0; s--) {
    const int R = z.radix[s];
    a.sub = len;
    len *= R;
    a.tws = z.n / len;
    a.items = a.nl * (z.n / R);
    if (s > 0) z_stage_any<1, false>(R, a);
    else z_last_any(R, a, o);
    __syncthreads();
  }
}
template <int R0, int R1>
__device__ __forceinline__ void z_forward(const ZPlan& z, ZStage a) {
  if constexpr (R0 == 0) {
    z_forward_any(z, a);
  } else {
    const float rl = __frcp_rn((float)a.nl);
    const int ps = a.ps;
#pragma unroll 1
    for (int q = threadIdx.x; q < a.nl * R1; q += blockDim.x) {
      int l;
      const int t = fdivmod(q, a.nl, rl, l);
      z_item<R0, -1, true, true>(z_line(a, l) + (uint32_t)(t * ps), (uint32_t)(R1 * ps), a.tw, t);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = threadIdx.x; q < a.nl * R0; q += blockDim.x) {
      int l;
      const int b = fdivmod(q, a.nl, rl, l);
      z_item<R1, -1, false, false>(z_line(a, l) + (uint32_t)(b * R1 * ps), (uint32_t)ps, a.tw, 0);
    }
    __syncthreads();
  }
}
template <int R0, int R1>
__device__ __forceinline__ void z_inverse(const ZPlan& z, ZStage a, const ZOut& o) {
  if constexpr (R0 == 0) {
    z_inverse_any(z, a, o);
  } else {
    const float rl = __frcp_rn((float)a.nl);
    const int ps = a.ps;
    a.tws = 1;
#pragma unroll 1
    for (int q = threadIdx.x; q < a.nl * R0; q += blockDim.x) {
      int l;
      const int b = fdivmod(q, a.nl, rl, l);
      z_item<R1, 1, false, false>(z_line(a, l) + (uint32_t)(b * R1 * ps), (uint32_t)ps, a.tw, 0);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = threadIdx.x; q < a.nl * R1; q += blockDim.x) {
      int l;
      const int t = fdivmod(q, a.nl, rl, l);
      z_last_item<R0, true>(a, o, l, t, (uint32_t)(R1 * ps), (size_t)R1 * o.kstride);
    }
    __syncthreads();
  }
}

// kz at position p after the forward stages
__device__ __forceinline__ int pencil_kz_dev(const ZPlan& z, int p) {
  int kz = 0, mul = 1, len = z.n;
  for (int s = 0; s < z.ns; s++) {
    len /= z.radix[s];
    const int d = p / len;
    p -= d * len;
    kz += mul * d;
    mul *= z.radix[s];
  }
  return kz;
}

// ------------------------------------------------------------------ per-bin algebra, eigen form

// A pair of bins between the posterior and the realisations: mu_post, and S_post as its real
// diagonal 00 11 22 and its entries 01 02 12.
struct PairPost {
  C2 mu[3];
  float2 sd[3];
  C2 so[3];
};

// am = A_l mu
__device__ __forceinline__ C2 a_mu(const ZParams& P, int l, const C2 (&m)[3]) {
  return c2_fma(P.A[l][2], m[2], c2_fma(P.A[l][1], m[1], c2_scale(m[0], P.A[l][0])));
}
// x - k y, the product rounded before the difference: residuals are differences of large numbers, and
// zpass.cuh forms them in this order too
__device__ __forceinline__ C2 c2_submul(C2 x, float kr, float ki, C2 y) {
  const float2 r = f2_fma(f2_dup(kr), y.r, f2_mul(f2_dup(-ki), y.i));
  const float2 i = f2_fma(f2_dup(kr), y.i, f2_mul(f2_dup(ki), y.r));
  return {f2_sub(x.r, r), f2_sub(x.i, i)};
}

// mu_post and S_post of the two bins of one z position from that position's row e (float4 groups
// at stride nzp, laid out as EigLayout: the angles' rows are streamed one at a time), and with
// RES the residuals in d.
template <int NTH, bool RES>
__device__ __forceinline__ void pair_posterior_eig(const ZParams& P, const float4* __restrict__ e, float2 lam,
                                                   float2 rho, const C2 (&mu)[3], C2 (&d)[NTH], PairPost& o) {
  constexpr int VP = pad4(2 * NTH), OKW = 0, OL = VP, OR = OL + pad4(NTH), RS = VP + 16;
  const int st = P.nzp;
  float Lm[pad4(NTH)];
  ldrow(Lm, e + (OL / 4) * st, st);
  {
    float kw[VP];
    ldrow(kw, e + (OKW / 4) * st, st);
    // d <- y = d - K mu, K = diag(kw) A
#pragma unroll
    for (int l = 0; l < NTH; l++) d[l] = c2_submul(d[l], kw[2 * l], kw[2 * l + 1], a_mu(P, l, mu));
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    o.mu[a] = mu[a];
    o.sd[a] = f2_mul(rho, f2_dup(P.pv[a]));
    o.so[a] = {f2_mul(rho, f2_dup(P.pv[3 + a])), make_float2(0.f, 0.f)};
  }
#pragma unroll
  for (int l = 0; l < NTH; l++) {
    // r_l = (V y)_l, s_l = r_l lam / (lam Lam_l + 1), w_l = lam^2 / (lam Lam_l + 1)
    float V[VP];
    ldrow(V, e + ((OR + l * RS) / 4) * st, st);
    float QH[16];
    ldrow(QH, e + ((OR + l * RS + VP) / 4) * st, st);
    const float* h = QH + 6;
    C2 r = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int m = 0; m < NTH; m++) {
      const float vr = V[2 * m], vi = V[2 * m + 1];
      r = {f2_fma(f2_dup(-vi), d[m].i, f2_fma(f2_dup(vr), d[m].r, r.r)),
           f2_fma(f2_dup(vi), d[m].r, f2_fma(f2_dup(vr), d[m].i, r.i))};
    }
    const float2 den = f2_fma(lam, f2_dup(Lm[l]), make_float2(1.f, 1.f));
    const float2 f = f2_mul(lam, make_float2(__frcp_rn(den.x), __frcp_rn(den.y)));
    const C2 sl = {f2_mul(r.r, f), f2_mul(r.i, f)};
    const float2 nw = f2_neg(f2_mul(lam, f));
    // mu_post += conj(Q_l.) s_l;  S_post -= w_l H_l, H_l = (|Q_l0|^2, |Q_l1|^2, |Q_l2|^2,
    // conj(Q_l0) Q_l1, conj(Q_l0) Q_l2, conj(Q_l1) Q_l2)
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float qr = QH[2 * a], qi = QH[2 * a + 1];
      o.mu[a] = {f2_fma(f2_dup(qi), sl.i, f2_fma(f2_dup(qr), sl.r, o.mu[a].r)),
                 f2_fma(f2_dup(-qi), sl.r, f2_fma(f2_dup(qr), sl.i, o.mu[a].i))};
      o.sd[a] = f2_fma(nw, f2_dup(h[a]), o.sd[a]);
      o.so[a] = {f2_fma(nw, f2_dup(h[3 + 2 * a]), o.so[a].r), f2_fma(nw, f2_dup(h[4 + 2 * a]), o.so[a].i)};
    }
  }
  // residual d - K mu_post = y - K (mu_post - mu) (the data spectrum itself where the row is zero:
  // kz not inverted)
  if (RES && P.keep_resid) {
    float kw[VP];
    ldrow(kw, e + (OKW / 4) * st, st);
    C2 dm[3];
#pragma unroll
    for (int a = 0; a < 3; a++) dm[a] = c2_sub(o.mu[a], mu[a]);
#pragma unroll
    for (int l = 0; l < NTH; l++) d[l] = c2_submul(d[l], kw[2 * l], kw[2 * l + 1], a_mu(P, l, dm));
  }
}

// lib_matrCholCpx(3) of both bins' S_post (simulate :1425-1443): chol_ref (pencil_common.cuh) on
// pairs.  L: sd holds the diagonal, so L10, L20, L21.  Returns bit u for a bin without a factor,
// whose entries stay S_post.
__device__ __forceinline__ int pair_factor(PairPost& o) {
  const float2 s11 = o.sd[1], s22 = o.sd[2], f = o.sd[0];
  const float2 i0 = make_float2(rsqrtf(f.x), rsqrtf(f.y));
  const float2 tol = f2_mul(f, f2_dup(1e-20f));
  const C2 l10 = {f2_mul(o.so[0].r, i0), f2_mul(f2_neg(o.so[0].i), i0)};
  const C2 l20 = {f2_mul(o.so[1].r, i0), f2_mul(f2_neg(o.so[1].i), i0)};
  const float2 r1 = f2_sub(s11, f2_fma(l10.i, l10.i, f2_mul(l10.r, l10.r)));
  const float2 i1 = make_float2(rsqrtf(r1.x), rsqrtf(r1.y));
  // a21 - L20 conj(L10), a21 = conj(S12)
  const float2 tr = f2_sub(o.so[2].r, f2_fma(l20.i, l10.i, f2_mul(l20.r, l10.r)));
  const float2 ti = f2_sub(f2_neg(o.so[2].i), f2_sub(f2_mul(l20.i, l10.r), f2_mul(l20.r, l10.i)));
  const C2 l21 = {f2_mul(tr, i1), f2_mul(ti, i1)};
  const float2 r2 = f2_sub(f2_sub(s22, f2_fma(l20.i, l20.i, f2_mul(l20.r, l20.r))),
                           f2_fma(l21.i, l21.i, f2_mul(l21.r, l21.r)));
  const float2 i2 = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const bool ok0 = f.x > 0.f && s11.x > tol.x && r1.x > tol.x && s22.x > tol.x && r2.x > tol.x;
  const bool ok1 = f.y > 0.f && s11.y > tol.y && r1.y > tol.y && s22.y > tol.y && r2.y > tol.y;
  const float2 d[3] = {f2_mul(f, i0), f2_mul(r1, i1), f2_mul(r2, i2)};
  const C2 lo[3] = {l10, l20, l21};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    if (ok0) {
      o.sd[a].x = d[a].x;
      o.so[a].r.x = lo[a].r.x;
      o.so[a].i.x = lo[a].i.x;
    }
    if (ok1) {
      o.sd[a].y = d[a].y;
      o.so[a].r.y = lo[a].r.y;
      o.so[a].i.y = lo[a].i.y;
    }
  }
  return (ok0 ? 0 : 1) | (ok1 ? 0 : 2);
}

// S_post = L L^H of the bins that have a factor (mask as pair_factor returned it).
__device__ __forceinline__ void pair_llh(float2 (&sd)[3], C2 (&so)[3], int fail) {
  const float2 l0 = sd[0], l1 = sd[1], l2 = sd[2];
  const C2 l10 = so[0], l20 = so[1], l21 = so[2];
  const float2 d[3] = {f2_mul(l0, l0), f2_fma(l10.r, l10.r, f2_fma(l10.i, l10.i, f2_mul(l1, l1))),
                       f2_fma(l20.r, l20.r,
                              f2_fma(l20.i, l20.i, f2_fma(l21.r, l21.r, f2_fma(l21.i, l21.i, f2_mul(l2, l2)))))};
  const C2 s[3] = {{f2_mul(l0, l10.r), f2_neg(f2_mul(l0, l10.i))},
                   {f2_mul(l0, l20.r), f2_neg(f2_mul(l0, l20.i))},
                   {f2_fma(l10.r, l20.r, f2_fma(l10.i, l20.i, f2_mul(l1, l21.r))),
                    f2_sub(f2_mul(l10.i, l20.r), f2_fma(l10.r, l20.i, f2_mul(l1, l21.i)))}};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    if (!(fail & 1)) {
      sd[a].x = d[a].x;
      so[a].r.x = s[a].r.x;
      so[a].i.x = s[a].i.x;
    }
    if (!(fail & 2)) {
      sd[a].y = d[a].y;
      so[a].r.y = s[a].r.y;
      so[a].i.y = s[a].i.y;
    }
  }
}

// ------------------------------------------------------------------ the kernel
//
// Shared memory: tw [nzp] (float2), the grid pointers of one batch of output lines (12), perm
// [nzp] (uint16: kz of a position; position of a kz in the Cholesky forms), then the tile, PS bytes per position.  With NP = W / 2 pairs:
//   slot s, pair q         16-byte word s NP + q
//   inputs                 data 0 .. nth-1, mean nth .. nth+2
//   after the per-bin step SB realisations' spectra 0 .. 3 SB - 1, mu_post 3 SB .. 3 SB + 2,
//                          S_post 01 02 12 (or L10 L20 L21) 3 SB + 3 .. 3 SB + 5
//   diagonal of S_post (L) words D NP + q: {00, 11} of the pair's first bin, then of its second;
//                          words D NP + NP + q / 2: 22 of the first bin at float q % 2, of the second
//                          at 2 + q % 2
// (D >= nth + 3 keeps the diagonal, which the threads of two pairs write, clear of the inputs; x-bins
// 2 m and 2 m + 1 share a complex line whatever W is, so W does not change the results).
enum PencilMode { kEig = 0, kChol = 1, kCholFp64 = 2 };

__device__ __forceinline__ void sts1(uint32_t a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void diag_put(uint32_t pos, const ZParams& P, int q, const float2 (&d)[3]) {
  const uint32_t w = pos + 16u * (uint32_t)(P.D * P.NP);
  sts4(w + 16u * (uint32_t)q, make_float4(d[0].x, d[1].x, d[0].y, d[1].y));
  const uint32_t x = w + 16u * (uint32_t)(P.NP + (q >> 1)) + 4u * (uint32_t)(q & 1);
  sts1(x, d[2].x);
  sts1(x + 8u, d[2].y);
  if (P.NP == 1) {   // no second pair in the word: its line is zero
    sts1(x + 4u, 0.f);
    sts1(x + 12u, 0.f);
  }
}
// ... of the pair's bin u alone
__device__ __forceinline__ void diag_put1(uint32_t pos, const ZParams& P, int q, int u, float d0, float d1, float d2) {
  const uint32_t w = pos + 16u * (uint32_t)(P.D * P.NP);
  sts2(w + 16u * (uint32_t)q + 8u * (uint32_t)u, make_float2(d0, d1));
  const uint32_t x = w + 16u * (uint32_t)(P.NP + (q >> 1)) + 4u * (uint32_t)(q & 1) + 8u * (uint32_t)u;
  sts1(x, d2);
  if (P.NP == 1) sts1(x + 4u, 0.f);
}
__device__ __forceinline__ void diag_get(uint32_t pos, const ZParams& P, int q, float2 (&d)[3]) {
  const uint32_t w = pos + 16u * (uint32_t)(P.D * P.NP);
  const float4 a = lds4(w + 16u * (uint32_t)q);
  const uint32_t x = w + 16u * (uint32_t)(P.NP + (q >> 1)) + 4u * (uint32_t)(q & 1);
  d[0] = make_float2(a.x, a.z);
  d[1] = make_float2(a.y, a.w);
  d[2] = make_float2(lds1(x), lds1(x + 8u));
}

template <int NTH, int MODE, int R0, int R1>
__global__ void __launch_bounds__(512, 1) k_pencil(const __grid_constant__ ZParams P) {
  extern __shared__ __align__(16) unsigned char smb[];
  __shared__ unsigned long long cnt[4];
  constexpr int GIN = NTH + 3;
  constexpr bool kResid = R0 != 0;   // residual spectra at the other lengths are zpass.cuh's
  const int NZ = P.nzp, NP = P.NP, lnp = P.logNP, W = 2 * NP, SB = P.SB, PS = P.PS;
  const int T = blockDim.x, tid = threadIdx.x;
  const uint32_t s_tw = smem_addr(smb), s_out = s_tw + 8u * (uint32_t)even_up_z(NZ), s_perm = s_out + 96u;
  const uint32_t tile = s_perm + 2u * (uint32_t)((NZ + 7) & ~7);
  const uint16_t* perm = reinterpret_cast<const uint16_t*>(smb + (s_perm - s_tw));
  unsigned long long* outp = reinterpret_cast<unsigned long long*>(smb + (s_out - s_tw));
  const int it = blockIdx.x % P.nIT, j = blockIdx.x / P.nIT;
  // x-offsets w in [wlo, nw) of the tile are bins i0 + w of the grid
  const int i0 = it * W - (P.vec ? (j * P.cnxp) & 1 : 0), wlo = i0 < 0 ? 1 : 0, nw = min(W, P.cnxp - i0);
  if (nw <= 0) return;   // a row without the early bin may need one tile less
  const size_t kstride = (size_t)P.nyp * P.cnxp;
  const size_t base = (size_t)j * P.cnxp + i0;

  dep_wait();
  dep_launch();
  // ---- inputs, natural kz order; x-bins beyond the grid are zero-filled
  for (int e = tid; e < NZ << lnp; e += T) {
    const int q = e & (NP - 1), w = 2 * q, k = e >> lnp;
    const bool in0 = w >= wlo && w < nw, in1 = w + 1 < nw;
    const size_t go = base + (size_t)k * kstride + w;
    const uint32_t sa = tile + (uint32_t)(k * PS) + 16u * (uint32_t)q;
    if (P.vec && in0 && in1) {
#pragma unroll
      for (int g = 0; g < GIN; g++)
        cp_async16(sa + 16u * (uint32_t)(g << lnp), (g < NTH ? P.data[g] : P.mean[g - NTH]) + go);
    } else {
#pragma unroll
      for (int g = 0; g < GIN; g++) {
        const float2* src = g < NTH ? P.data[g] : P.mean[g - NTH];
        const uint32_t d = sa + 16u * (uint32_t)(g << lnp);
        cp_async8_zfill(d, src + (in0 ? go : 0), in0);
        cp_async8_zfill(d + 8u, src + (in1 ? go + 1 : 0), in1);
      }
    }
  }
  cp_async_commit();
  if (tid < 4) cnt[tid] = 0;
  for (int t = tid; t < NZ; t += T) {
    sts2(s_tw + 8u * (uint32_t)t, __ldg(P.twz + t));
    const int kz = pencil_kz_dev(P.z, t);
    const_cast<uint16_t*>(perm)[MODE == kEig ? t : kz] = (uint16_t)(MODE == kEig ? kz : t);
  }
  cp_async_wait_0();
  __syncthreads();
  ZStage zs;
  zs.base = tile;
  zs.tw = s_tw;
  zs.ps = PS;
  zs.nl = GIN << lnp;
  zs.split = zs.nl;
  zs.gap = 0;
  z_forward<R0, R1>(P.z, zs);
  // a NaN or Inf in any input grid reaches every bin through the transforms
  // (read by the thread whose per-bin step takes that bin first)
  if (tid == (MODE == kEig ? 0 : wlo) && P.counters) {
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < GIN; g++) {
      const float4 v = lds4(tile + 16u * (uint32_t)(g << lnp));
      s += wlo ? fabsf(v.y) + fabsf(v.w) : fabsf(v.x) + fabsf(v.z);
    }
    if (!isfinite(s)) atomicAdd(P.counters + 4, 1ull);
  }

  // ---- per-bin posterior.  The positions of neighbouring threads are p and p ^ 3 swapped within
  //      fours where that puts their words on different banks (P.swz)
  const int items = NZ << lnp;
  const uint32_t s_post = 16u * (uint32_t)((3 * SB) << lnp);   // byte offset of mu_post in a position
  unsigned long long n_zero_bins = 0, n_inv = 0, n_fail = 0, n_fp64 = 0;
  unsigned int failed = 0;                                    // two bits per item of this thread
  // Position and kz of the m-th round.  The eigen form takes the positions in order; the Cholesky forms the
  // kz in order: the kz that are not inverted and the bins that FP64 does again come in runs, which whole
  // warps then skip or take, where digit-reversed every warp holds a few (200x216x200, prior grids: 0.80 -> 0.74 ms,
  // with FP64 0.82 -> 0.75; 60x50x128, FP64: 74 -> 62 us).
  auto locate = [&](int m, int& p, int& kz) {
    if constexpr (MODE == kEig) {
      p = P.swz ? (m & ~3) | ((m & 1) << 1) | ((m >> 1) & 1) : m;
      kz = perm[p];
    } else {
      kz = m;
      p = perm[m];
    }
  };
  if constexpr (MODE != kEig) {
    // The Cholesky forms: a bin, not a pair, per thread and round.  A factorisation is a serial chain, longer by
    // several times where it is done again in FP64, and on a small block the chains of one tile are the time
    // of the pass (28x27x45, 5 angles, FP64: 73 us with a pair's two chains in one thread, 52 so).  Lane u of a
    // pair's words is its bin u: the two threads of a pair share words, but no float.
#pragma unroll 1
    for (int b = tid; b < 2 * items; b += T) {
      const int u = b & 1, q = (b >> 1) & (NP - 1), w = 2 * q + u;
      int p, kz;
      locate(b >> (1 + lnp), p, kz);
      const uint32_t pos = tile + (uint32_t)(p * PS), sl = pos + 16u * (uint32_t)q + 4u * (uint32_t)u;
      const bool in = w >= wlo && w < nw;
      const size_t gi = base + (size_t)kz * kstride + w;
      float2 m1[3], d1[NTH];
#pragma unroll
      for (int l = 0; l < NTH; l++) {
        const uint32_t x = sl + 16u * (uint32_t)(l << lnp);
        d1[l] = make_float2(lds1(x), lds1(x + 8u));
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const uint32_t x = sl + 16u * (uint32_t)((NTH + a) << lnp);
        m1[a] = make_float2(lds1(x), lds1(x + 8u));
      }
      float S[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, lam = 0.f, rho = 0.f;
      if (in) {
        if (P.separable) {
          const float2 cx = __ldg(P.cxy + base + w), c_t = __ldg(P.ct + kz);
          rho = fabsf(cx.x * c_t.x - cx.y * c_t.y);
#pragma unroll
          for (int c = 0; c < 6; c++) S[c] = P.pv[c] * rho;
          lam = fabsf(cx.x);
        } else {
          // getNextParameterCovariance: |Re/pv| pv (no division when pv == 0); a base prior's
          // pairs share |Re/pv| of the one spectrum transformed (pv[0] != 0)
          if (P.base_prior) {
            const float r0 = fabsf(P.cov[0][gi].x / P.pv[0]);
#pragma unroll
            for (int c = 0; c < 6; c++) S[c] = r0 * P.pv[c];
          } else {
#pragma unroll
            for (int c = 0; c < 6; c++) {
              float re = P.cov[c][gi].x;
              const float pv = P.pv[c];
              if (pv != 0.f) re = re / pv;
              S[c] = fabsf(re) * pv;
            }
          }
          lam = fabsf(P.errspec[gi].x);
        }
      }
      BinOut bo;
      bool ok = false;
      if (in && P.kz.inv[kz] != 0) {
        n_inv++;
        ok = P.septab ? bin_posterior<NTH, true>(P, kz, S, lam, rho, m1, d1, bo)
                      : bin_posterior<NTH, false>(P, kz, S, lam, rho, m1, d1, bo);
        if constexpr (MODE == kCholFp64) {
          if (ok) {
            float ratio = 1.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
              if (S[a] > 0.f) ratio = fminf(ratio, bo.sp[a].x / S[a]);
            if (bo.cond > P.fp64_threshold || ratio * P.fp64_threshold < 1.f) {
              // the data are still in their slots: restart from them
              float2 d64[NTH];
#pragma unroll
              for (int l = 0; l < NTH; l++) {
                const uint32_t x = sl + 16u * (uint32_t)(l << lnp);
                d64[l] = make_float2(lds1(x), lds1(x + 8u));
              }
              if (bin_posterior_fp64<NTH>(P, kz, S, lam, m1, d64, bo)) {
                n_fp64++;
#pragma unroll
                for (int l = 0; l < NTH; l++) d1[l] = d64[l];
              }
            }
          }
        }
        if (!ok) n_fail++;
      }
      if (!ok) {
#pragma unroll
        for (int a = 0; a < 3; a++) bo.mu[a] = m1[a];
#pragma unroll
        for (int c = 0; c < 6; c++) bo.sp[c] = make_float2(S[c], 0.f);
      }
      if constexpr (kResid)
        if (P.keep_resid && in) {
#pragma unroll
          for (int l = 0; l < NTH; l++) P.data[l][gi] = d1[l];
        }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const uint32_t xm = sl + s_post + 16u * (uint32_t)(a << lnp), xs = sl + s_post + 16u * (uint32_t)((3 + a) << lnp);
        sts1(xm, bo.mu[a].x);
        sts1(xm + 8u, bo.mu[a].y);
        sts1(xs, bo.sp[3 + a].x);
        sts1(xs + 8u, bo.sp[3 + a].y);
      }
      diag_put1(pos, P, q, u, bo.sp[0].x, bo.sp[1].x, bo.sp[2].x);
    }
    __syncthreads();
  }
  // The eigen form, two bins a thread.  Then, in every form, S_post is factored once for all realisations; the
  // covariance output is rebuilt as L L^H
  if (MODE == kEig || P.nsim > 0) {
    int n = 0;
#pragma unroll 1
    for (int b = tid; b < items; b += T, n++) {
      const int q = b & (NP - 1);
      int p, kz;
      locate(b >> lnp, p, kz);
      const uint32_t pos = tile + (uint32_t)(p * PS), sl = pos + 16u * (uint32_t)q, so = sl + s_post;
      const bool in0 = 2 * q >= wlo && 2 * q < nw, in1 = 2 * q + 1 < nw;
      PairPost o;
      if constexpr (MODE == kEig) {
        C2 mu[3], d[NTH];
#pragma unroll
        for (int l = 0; l < NTH; l++) d[l] = lds_c2(sl + 16u * (uint32_t)(l << lnp));
#pragma unroll
        for (int a = 0; a < 3; a++) mu[a] = lds_c2(sl + 16u * (uint32_t)((NTH + a) << lnp));
        float2 lam, rho;
        {
          const float ctk = __ldg(P.ct + kz).x;
          const float2* cx = P.cxy + base + 2 * q;
          const float c0 = in0 ? __ldg(cx).x : 0.f, c1 = in1 ? __ldg(cx + 1).x : 0.f;
          lam = make_float2(fabsf(c0), fabsf(c1));
          rho = make_float2(fabsf(c0 * ctk), fabsf(c1 * ctk));
        }
        pair_posterior_eig<NTH, kResid>(P, P.eig + p, lam, rho, mu, d, o);
        if constexpr (kResid)
          if (P.keep_resid) {
            const size_t gidx = base + (size_t)kz * kstride + 2 * q;
#pragma unroll
            for (int l = 0; l < NTH; l++) {
              if (in0) P.data[l][gidx] = make_float2(d[l].r.x, d[l].i.x);
              if (in1) P.data[l][gidx + 1] = make_float2(d[l].r.y, d[l].i.y);
            }
          }
      } else {
        diag_get(pos, P, q, o.sd);
#pragma unroll
        for (int a = 0; a < 3; a++) o.so[a] = lds_c2(so + 16u * (uint32_t)((3 + a) << lnp));
      }
      if (P.nsim > 0) {
        const int fail = pair_factor(o);
        failed |= (unsigned int)fail << (2 * n);
        if ((fail & 1) && in0) n_zero_bins++;
        if ((fail & 2) && in1) n_zero_bins++;
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        if constexpr (MODE == kEig) sts_c2(so + 16u * (uint32_t)(a << lnp), o.mu[a]);
        sts_c2(so + 16u * (uint32_t)((3 + a) << lnp), o.so[a]);
      }
      diag_put(pos, P, q, o.sd);
    }
  }
  ZOut zo;
  zo.out = s_out;
  zo.base = base;
  zo.kstride = kstride;
  zo.wlo = wlo;
  zo.nw = nw;
  zo.logNP = lnp;
  zo.vec = P.vec;
  __syncthreads();

  // ---- realisations, the mean added in the spectral domain; SB share one transform
#pragma unroll 1
  for (int s0 = 0; s0 < P.nsim; s0 += SB) {
    const int nb = min(SB, P.nsim - s0);
    const bool last = s0 + nb == P.nsim;
    if (tid < 3 * nb) outp[tid] = (unsigned long long)(uintptr_t)P.sim[3 * s0 + tid];
    int n = 0;
#pragma unroll 1
    for (int b = tid; b < items; b += T, n++) {
      const int q = b & (NP - 1);
      int p, kz;
      locate(b >> lnp, p, kz);
      const uint32_t pos = tile + (uint32_t)(p * PS), sl = pos + 16u * (uint32_t)q, so = sl + s_post;
      const int fail = (failed >> (2 * n)) & 3;
      float2 ld[3];
      diag_get(pos, P, q, ld);
      C2 lo[3], mu[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        mu[a] = lds_c2(so + 16u * (uint32_t)(a << lnp));
        lo[a] = lds_c2(so + 16u * (uint32_t)((3 + a) << lnp));
      }
#pragma unroll 1
      for (int sb = 0; sb < nb; sb++) {
        C2 z[3];
        if (P.host_noise) {
          float2 za[3], zb[3];
          {
            const size_t gidx = base + (size_t)kz * kstride + 2 * q;
            const bool in0 = 2 * q >= wlo && 2 * q < nw, in1 = 2 * q + 1 < nw;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              za[c] = in0 ? P.noise[3 * (s0 + sb) + c][gidx] : make_float2(0.f, 0.f);
              zb[c] = in1 ? P.noise[3 * (s0 + sb) + c][gidx + 1] : make_float2(0.f, 0.f);
            }
          }
#pragma unroll
          for (int c = 0; c < 3; c++) z[c] = {make_float2(za[c].x, zb[c].x), make_float2(za[c].y, zb[c].y)};
        } else {
          pair_noise(P, s0 + sb, i0 + 2 * q, j, kz, z);
        }
        // L z: rows (l0), (L10, l1), (L20, L21, l2)
        C2 x[3];
#pragma unroll
        for (int a = 0; a < 3; a++) x[a] = {f2_mul(ld[a], z[a].r), f2_mul(ld[a], z[a].i)};
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const int r = a == 0 ? 1 : 2, c = a == 2 ? 1 : 0;
          x[r] = {f2_sub(f2_fma(lo[a].r, z[c].r, x[r].r), f2_mul(lo[a].i, z[c].i)),
                  f2_fma(lo[a].r, z[c].i, f2_fma(lo[a].i, z[c].r, x[r].i))};
        }
#pragma unroll
        for (int a = 0; a < 3; a++) {
          if (fail & 1) x[a].r.x = x[a].i.x = 0.f;
          if (fail & 2) x[a].r.y = x[a].i.y = 0.f;
          sts_c2(sl + 16u * (uint32_t)((3 * sb + a) << lnp), c2_add(mu[a], x[a]));
        }
      }
      if (last) {
        pair_llh(ld, lo, fail);
#pragma unroll
        for (int a = 0; a < 3; a++) sts_c2(so + 16u * (uint32_t)((3 + a) << lnp), lo[a]);
        diag_put(pos, P, q, ld);
      }
    }
    __syncthreads();
    zs.nl = zs.split = (3 * nb) << lnp;
    z_inverse<R0, R1>(P.z, zs, zo);
  }

  // ---- inverse z transform of the posterior mean and covariance (unless it stays spectral)
  zs.base = tile + s_post;
  if (P.cov_spectral) {
    if (tid < 3) outp[tid] = (unsigned long long)(uintptr_t)P.mean[tid];
    for (int b = tid; b < items; b += T) {
      const int q = b & (NP - 1);
      int p, kz;
      locate(b >> lnp, p, kz);
      const uint32_t pos = tile + (uint32_t)(p * PS), so = pos + 16u * (uint32_t)q + s_post;
      const bool in0 = 2 * q >= wlo && 2 * q < nw, in1 = 2 * q + 1 < nw;
      const size_t gidx = base + (size_t)kz * kstride + 2 * q;
      float2 sd[3];
      diag_get(pos, P, q, sd);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const C2 s = lds_c2(so + 16u * (uint32_t)((3 + a) << lnp));
        if (in0) {
          P.cov[a][gidx] = make_float2(sd[a].x, 0.f);
          P.cov[3 + a][gidx] = make_float2(s.r.x, s.i.x);
        }
        if (in1) {
          P.cov[a][gidx + 1] = make_float2(sd[a].y, 0.f);
          P.cov[3 + a][gidx + 1] = make_float2(s.r.y, s.i.y);
        }
      }
    }
    zs.nl = zs.split = 3 << lnp;
    __syncthreads();
    z_inverse<R0, R1>(P.z, zs, zo);
  } else {
    if (tid < 6) outp[tid] = (unsigned long long)(uintptr_t)(tid < 3 ? P.mean[tid] : P.cov[tid]);
    const int ndl = NP + ((NP + 1) >> 1);               // words of the diagonal
    zs.split = 6 << lnp;
    zs.nl = zs.split + ndl;
    zs.gap = 16 * ((P.D - 3 * SB - 6) << lnp);
    __syncthreads();
    z_inverse<R0, R1>(P.z, zs, zo);
    // the diagonal's lines x = S_A + i S_B (S real spectra): S_A(z) = (x(z) + conj x(-z)) / 2,
    // S_B(z) = (x(z) - conj x(-z)) / 2i
    const int half = NZ / 2 + 1;
    const float rd = __frcp_rn((float)ndl);
    for (int e = tid; e < ndl * half; e += T) {
      int l;
      const int z = fdivmod(e, ndl, rd, l), zm = z == 0 ? 0 : NZ - z;
      const uint32_t wd = tile + 16u * (uint32_t)((P.D << lnp) + l);
      const float4 x = lds4(wd + (uint32_t)(z * PS)), y = lds4(wd + (uint32_t)(zm * PS));
#pragma unroll
      for (int h = 0; h < 2; h++) {
        // complex line h of the word: entry 00 (h = 0) or 11 of pair l, or 22 of pair 2 (l - NP) + h
        const int c = l < NP ? h : 2, q = l < NP ? l : 2 * (l - NP) + h, w = 2 * q;
        if (q >= NP) continue;
        const float xr = h ? x.y : x.x, xi = h ? x.w : x.z, yr = h ? y.y : y.x, yi = h ? y.w : y.z;
        const float2 A = make_float2(0.5f * (xr + yr), 0.5f * (xi - yi));
        const float2 B = make_float2(0.5f * (xi + yi), 0.5f * (yr - xr));
        const bool in0 = w >= wlo && w < nw, in1 = w + 1 < nw;
        float2* g = P.cov[c] + base + w;
        float2 *gz = g + (size_t)z * kstride, *gm = g + (size_t)zm * kstride;
        if (P.vec && in0 && in1) {
          *reinterpret_cast<float4*>(gz) = make_float4(A.x, A.y, B.x, B.y);
          if (zm != z) *reinterpret_cast<float4*>(gm) = make_float4(A.x, -A.y, B.x, -B.y);
        } else {
          if (in0) {
            gz[0] = A;
            if (zm != z) gm[0] = make_float2(A.x, -A.y);
          }
          if (in1) {
            gz[1] = B;
            if (zm != z) gm[1] = make_float2(B.x, -B.y);
          }
        }
      }
    }
  }

  // counters
  unsigned long long n_zero = n_zero_bins * (unsigned long long)P.nsim;
  for (int off = 16; off > 0; off >>= 1) {
    n_zero += __shfl_down_sync(0xffffffffu, n_zero, off);
    if (MODE != kEig) {
      n_inv += __shfl_down_sync(0xffffffffu, n_inv, off);
      n_fail += __shfl_down_sync(0xffffffffu, n_fail, off);
      n_fp64 += __shfl_down_sync(0xffffffffu, n_fp64, off);
    }
  }
  if ((tid & 31) == 0) {
    if (n_zero) atomicAdd(&cnt[2], n_zero);
    if (MODE != kEig) {
      atomicAdd(&cnt[0], n_inv);
      atomicAdd(&cnt[1], n_fail);
      atomicAdd(&cnt[3], n_fp64);
    }
  }
  __syncthreads();
  if (tid == 0 && P.counters) {
    // eigen form: inverted bins per tile column from the host's count of inverted kz
    atomicAdd(P.counters + 0, MODE == kEig ? (unsigned long long)P.n_inv_rows * (unsigned long long)(nw - wlo) : cnt[0]);
    if (cnt[1]) atomicAdd(P.counters + 1, cnt[1]);
    if (cnt[2]) atomicAdd(P.counters + 2, cnt[2]);
    if (cnt[3]) atomicAdd(P.counters + 3, cnt[3]);
  }
}

// ------------------------------------------------------------------ launch templates

template <int NTH, int MODE, int R0, int R1>
inline cudaError_t launch_pencil_t(const ZParams& zp, int threads, cudaStream_t st) {
  const size_t smem = pencil_smem_bytes(zp.W, zp.nzp, zp.nth, zp.SB);
  auto fn = k_pencil<NTH, MODE, R0, R1>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const size_t bytes = sizeof(float2) * (size_t)(12 + zp.nth + 3 * zp.nsim) * zp.cnxp * zp.nyp * zp.nzp;
  return launch_dep(bytes, fn, dim3((unsigned)(zp.nIT * zp.nyp)), threads, smem, st, zp);
}
// the lengths whose split is inlined (pencil_plan gives the same)
template <int NTH, int MODE>
inline cudaError_t launch_pencil_z(const ZParams& zp, int threads, cudaStream_t st) {
  switch (zp.nzp) {
#define CRAVA_CASE(N, R0, R1) \
  case N: return launch_pencil_t<NTH, MODE, R0, R1>(zp, threads, st);
    CRAVA_Z_INLINED(CRAVA_CASE)
#undef CRAVA_CASE
    default: return launch_pencil_t<NTH, MODE, 0, 0>(zp, threads, st);
  }
}
// FP64 re-factorisation or none
template <int NTH>
inline cudaError_t launch_pencil_chol(const ZParams& zp, int threads, cudaStream_t st) {
  return zp.fp64_threshold > 0.f ? launch_pencil_z<NTH, kCholFp64>(zp, threads, st)
                                 : launch_pencil_z<NTH, kChol>(zp, threads, st);
}

// launchers by angle count: the eigen form in pencil_n12.cu .. pencil_n78.cu, the Cholesky forms in
// pencil_c12.cu .. pencil_c78.cu.  The units compile side by side, and a process loads the whole of one at its first
// launch: with the forms in one unit, a process's first job took 31 ms at 540x540x256 and 28 at 250x250x200, apart 21 and 15.
cudaError_t launch_pencil_n12(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_n34(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_n56(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_n78(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_c12(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_c34(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_c56(const ZParams& zp, int threads, cudaStream_t st);
cudaError_t launch_pencil_c78(const ZParams& zp, int threads, cudaStream_t st);

}  // namespace crava

// Four-step transform kernels and their launch templates for the lengths of the size table
// in fft4.cu (sm_100a): the
// same transforms as k_x_r2c / k_x_c2r / k_line_fft (kernels.cu), with each line done in
// two register-codelet passes (fft2.cuh) instead of one shared-memory stage per radix.
//
//   k_line4<N,DIR>      W columns of one strided line set, in pairs: global -> first stage -> shared (->
//                       middle stage) -> last stage -> global; k_line4s<N1,N2,DIR> the same one by one
//   k_xr2c4<N1,N2>      rows of even nxp, h = nxp/2 = N1 N2: global -> shared -> pass 1 -> shared
//                       -> pass 2 and split -> shared -> global
//   k_xc2r4<N1,N2>      global -> shared -> merge and pass 1 -> shared -> pass 2 -> shared -> global
//   k_xr2c4o, k_xc2r4o  the same for odd nxp = N1 N2, two rows per complex line
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdlib>

#include "fft_pair.cuh"
#include "kernels.cuh"

namespace crava {

// shared layout of the kernels: n twiddles (rounded up to an even count, so that what follows starts on
// 16 bytes), the tile or the staged rows, the exchange buffer of the scalar row passes
constexpr int even_up(int n) { return (n + 1) & ~1; }

// ------------------------------------------------------------------ strided lines
//
// W columns (NP = W / 2 pairs of columns q, q + NP, C2 of fft_pair.cuh) of n = R0 R1 R2 points in two
// (R2 = 1) or three stages: the first reads global memory and leaves its results in the tile, the last
// stores to global memory in natural order.  With N1 = R1 R2 the decimation-in-frequency stages
// are
//   stage 0, item t < N1         x[t + N1 m] -> DFT_R0 -> w^(t k0)          at k0 N1 + t
//   stage 1, item (k0, t < R2)   at k0 N1 + t + R2 m -> DFT_R1 -> w^(R0 t k1)  at k0 N1 + k1 R2 + t
//   last stage, item b           at b R + m -> DFT_R -> X[rev(b) + (n / R) k]
// rev(b) = k0 + R0 k1 for b = k0 R1 + k1.  Radices of 16 at most keep a pair's data in 64 registers.
//
// Tile word (position p, pair q) at 16 (p NP + q) bytes: 8 pairs, a whole 128-byte line of banks.
struct ColSplit {
  int r0, r1, r2;
};
constexpr ColSplit col_split(int n) {
  for (int a = 2; a <= 16; a++)
    if (n % a == 0 && n / a <= a) return {a, n / a, 1};          // smallest larger factor
  for (int top = 2; top <= 32; top++)
    for (int a = top; a >= 2; a--) {
      if (n % a) continue;
      for (int b = a; b >= 2; b--)
        if ((n / a) % b == 0 && n / a / b <= b) return {a, b, n / a / b};
    }
  return {0, 0, 0};
}

template <int R, int DIR>
__device__ __forceinline__ void col_twiddle(C2 (&v)[R], const float2* tw, int step) {
#pragma unroll
  for (int k = 1; k < R; k++) {
    const float2 w = tw[step * k];
    v[k] = c2_mul(v[k], w.x, DIR < 0 ? w.y : -w.y);
  }
}

template <int N, int DIR>
__global__ void __launch_bounds__(256, col_split(N).r0 <= 10 ? 4 : col_split(N).r0 <= 12 ? 3 : 2) k_line4(const __grid_constant__ GridSet gs, int ni, size_t pstride,
                                               size_t ostride, int lnp, int nIT, const float2* __restrict__ twg) {
  constexpr ColSplit S = col_split(N);
  constexpr int R0 = S.r0, R1 = S.r1, R2 = S.r2, N1 = R1 * R2, RL = R2 > 1 ? R2 : R1;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  const uint32_t Y = smem_addr(sm + even_up(N));
  const int T = blockDim.x, tid = threadIdx.x, NP = 1 << lnp, W = 2 * NP;
  const int it = blockIdx.x % nIT, o = blockIdx.x / nIT;
  const int i0 = it * W, nw = min(W, ni - i0);
  float2* g = reinterpret_cast<float2*>(gs.p[blockIdx.y]) + (size_t)o * ostride + i0;
  const uint32_t ps = 16u << lnp;
  dep_wait();
  dep_launch();
  for (int t = tid; t < N; t += T) tw[t] = twg[t];
  bool first = true;
#pragma unroll 1
  for (int e = tid; e < NP * N1 || first; e += T) {
    const int q = e & (NP - 1), t = e >> lnp;
    const bool on = e < NP * N1, in0 = on && q < nw, in1 = on && q + NP < nw;
    C2 v[R0];
    {
      const float2* src = g + (size_t)t * pstride + q;
      const size_t st = (size_t)N1 * pstride;
#pragma unroll
      for (int m = 0; m < R0; m++, src += st) {
        const float2 a = in0 ? src[0] : make_float2(0.f, 0.f), b = in1 ? src[NP] : make_float2(0.f, 0.f);
        v[m] = {make_float2(a.x, b.x), make_float2(a.y, b.y)};
      }
    }
    DftP<R0, DIR>::run(v);
    if (first) {          // the table, staged behind the loads
      __syncthreads();
      first = false;
    }
    if (!on) break;
    col_twiddle<R0, DIR>(v, tw, t);
    const uint32_t y = Y + (uint32_t)t * ps + 16u * (uint32_t)q;
#pragma unroll
    for (int k = 0; k < R0; k++) sts_c2(y + (uint32_t)(k * N1) * ps, v[k]);
  }
  __syncthreads();
  if constexpr (R2 > 1) {
#pragma unroll 1
    for (int e = tid; e < NP * R0 * R2; e += T) {
      const int q = e & (NP - 1), j = e >> lnp, k0 = j / R2, t = j - k0 * R2;
      const uint32_t y = Y + (uint32_t)(k0 * N1 + t) * ps + 16u * (uint32_t)q;
      C2 v[R1];
#pragma unroll
      for (int m = 0; m < R1; m++) v[m] = lds_c2(y + (uint32_t)(m * R2) * ps);
      DftP<R1, DIR>::run(v);
      col_twiddle<R1, DIR>(v, tw, R0 * t);
#pragma unroll
      for (int k = 0; k < R1; k++) sts_c2(y + (uint32_t)(k * R2) * ps, v[k]);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int e = tid; e < NP * (N / RL); e += T) {
    const int q = e & (NP - 1), b = e >> lnp;
    const uint32_t y = Y + (uint32_t)(b * RL) * ps + 16u * (uint32_t)q;
    C2 v[RL];
#pragma unroll
    for (int m = 0; m < RL; m++) v[m] = lds_c2(y + (uint32_t)m * ps);
    DftP<RL, DIR>::run(v);
    const int k0 = R2 > 1 ? b / R1 : b, rev = R2 > 1 ? k0 + R0 * (b - k0 * R1) : b;
    float2* dst = g + (size_t)rev * pstride + q;
    const size_t st = (size_t)(N / RL) * pstride;
    if (q + NP < nw) {
#pragma unroll
      for (int k = 0; k < RL; k++, dst += st) {
        dst[0] = make_float2(v[k].r.x, v[k].i.x);
        dst[NP] = make_float2(v[k].r.y, v[k].i.y);
      }
    } else if (q < nw) {
#pragma unroll
      for (int k = 0; k < RL; k++, dst += st) dst[0] = make_float2(v[k].r.x, v[k].i.x);
    }
  }
}

// The scalar two-pass form of the other lengths (line4 below says which), one column an item.
//
// One tile of W columns (nw of them valid) of the lines through g: point p of column w at
// g[p pstride + w], read from src[p spstride + w] (g itself, or a staged copy of the tile in
// shared memory).  Shared layout of the W lines: element (w, p = t + N2 m) at
// p W + w + m SK, with SK chosen so that the pass-2 reads of neighbouring k2 fall on
// disjoint banks.  Needs tw (the length-N table) in shared memory; ends with a barrier.
template <int N1, int N2, int DIR>
__device__ __forceinline__ void line4_tile(const float2* srcb, size_t spstride, float2* g, int nw, size_t pstride,
                                           int W, int lw, int SK, const float2* tw, float2* Y) {
  const int T = blockDim.x, tid = threadIdx.x;
  const size_t mstride = (size_t)N2 * spstride;
  const int mpitch = N2 * W + SK;
  for (int q = tid; q < W * N2; q += T) {
    const int w = q & (W - 1), t = q >> lw;
    const bool ok = w < nw;
    const float2* src = srcb + (size_t)t * spstride + w;
    float2* y = Y + t * W + w;
    four_step_pass1<N1, N2, DIR>(
        t, tw, [&](int, int m) { return ok ? src[m * mstride] : make_float2(0.f, 0.f); },
        [&](int, int k2, float2 v) { y[k2 * mpitch] = v; });
  }
  __syncthreads();
  for (int q = tid; q < W * N1; q += T) {
    const int w = q & (W - 1), k2 = q >> lw;
    const float2* y = Y + k2 * mpitch + w;
    float2 v[N2];
    four_step_pass2<N1, N2, DIR>(k2, [&](int, int t) { return y[t * W]; }, v);
    if (w < nw) {
      float2* dst = g + (size_t)k2 * pstride + w;
#pragma unroll
      for (int k1 = 0; k1 < N2; k1++) dst[(size_t)k1 * N1 * pstride] = v[k1];
    }
  }
  __syncthreads();
}

template <int N1, int N2>
constexpr size_t line4_smem(int W, int SK) {
  return sizeof(float2) * ((size_t)W * N1 * N2 + (size_t)N1 * SK);
}

// Forward instances bounded at 256 threads (the register allocation the forward passes were
// tuned with), inverse ones at 512 (a CTA may take one pass in a single round).
template <int N1, int N2, int DIR>
__global__ void __launch_bounds__(DIR > 0 ? 512 : 256) k_line4s(const __grid_constant__ GridSet gs, int ni, size_t pstride,
                                               size_t ostride, int W, int lw, int nIT, int SK,
                                               const float2* __restrict__ twg, int pf) {
  constexpr int N = N1 * N2;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  dep_wait();
  dep_launch();
  for (int t = threadIdx.x; t < N; t += blockDim.x) tw[t] = twg[t];
  const int it = blockIdx.x % nIT, o = blockIdx.x / nIT;
  const int i0 = it * W, nw = min(W, ni - i0);
  float2* g = reinterpret_cast<float2*>(gs.p[blockIdx.y]) + (size_t)o * ostride + i0;
  // pf > 0: the cache lines of the tile pf block indices on (x fastest) go to L2
  if (pf > 0) {
    const int tn = blockIdx.y * gridDim.x + blockIdx.x + pf;
    if (tn < (int)(gridDim.x * gridDim.y)) {
      const int gy = tn / gridDim.x, gx = tn - gy * gridDim.x;
      const int itn = gx % nIT, on = gx / nIT;
      const int nwn = min(W, ni - itn * W);
      const float2* gn = reinterpret_cast<const float2*>(gs.p[gy]) + (size_t)on * ostride + itn * W;
      for (int q = threadIdx.x; q < 2 * N; q += blockDim.x) {
        const float2* row = gn + (size_t)(q >> 1) * pstride;
        l2_prefetch_line((q & 1) ? (const void*)(row + nwn - 1) : (const void*)row);
      }
    }
  }
  __syncthreads();
  line4_tile<N1, N2, DIR>(g, pstride, g, nw, pstride, W, lw, SK, tw, sm + N);
}

// ------------------------------------------------------------------ rows, even nxp
//
// Row r of a unit in shared memory at r * PITCH; pass-1 position t + N2 m at
// t + m (N2 + SK) with SK = 1 for even N2 (odd stride for the pass-2 reads).
template <int N1, int N2>
struct RowLayout {
  static constexpr int H = N1 * N2;
  static constexpr int SK = (N2 % 2 == 0) ? 1 : 0;
  static constexpr int PITCH = H + N1 * SK;
  static __device__ __forceinline__ int pad(int t, int m) { return t + m * (N2 + SK); }
};

// nr rows, even nxp: src rows (h complex values x[2m] + i x[2m+1] each, row pitch h + 1) to
// the scaled half spectra in dst (may equal src).  The split step as k_x_r2c (kernels.cu),
// done in registers: output k = k2 + N1 k1 of pass-2 item k2 has its mirror h - k in item
// (N1 - k2) mod N1, so one thread takes both items of a pair (k2 <= N1 / 2) and forms every
// X[k], X[h-k] from the two DFTs it holds.  Needs tw (length h) and twh (e^{-2 pi i k / nxp},
// k < h) in shared memory; Z: rpc * PITCH.  Ends with a barrier.
template <int N1, int N2>
__device__ __forceinline__ void xr2c4_rows(const float2* src, float2* dst, int nr, float scale, const float2* tw,
                                           const float2* twh, float2* Z) {
  using L = RowLayout<N1, N2>;
  constexpr int H = L::H, PITCH = L::PITCH;
  constexpr int CN = H + 1, NPI = N1 / 2 + 1;
  const int T = blockDim.x, tid = threadIdx.x;
  for (int q = tid; q < nr * N2; q += T) {
    const int r = q / N2, t = q - r * N2;
    const float2* x = src + (size_t)r * CN + t;
    float2* z = Z + r * PITCH;
    four_step_pass1<N1, N2, -1>(
        t, tw, [&](int, int m) { return x[m * N2]; }, [&](int, int k2, float2 v) { z[L::pad(t, k2)] = v; });
  }
  __syncthreads();
  for (int q = tid; q < nr * NPI; q += T) {
    const int r = q / NPI, a = q - r * NPI;        // item a and its mirror item b
    const int b = a == 0 ? 0 : N1 - a;
    const float2* z = Z + r * PITCH;
    float2 va[N2], vb[N2];
    four_step_pass2<N1, N2, -1>(a, [&](int k, int t) { return z[L::pad(t, k)]; }, va);
    if (b != a) four_step_pass2<N1, N2, -1>(b, [&](int k, int t) { return z[L::pad(t, k)]; }, vb);
    float2* X = dst + (size_t)r * CN;
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) {
      const int k = a + N1 * k1;
      if (k == 0) {
        const float2 z0 = va[0];
        X[0] = make_float2(scale * (z0.x + z0.y), 0.f);
        X[H] = make_float2(scale * (z0.x - z0.y), 0.f);
        continue;
      }
      // z[h - k]: item b's output N2 - 1 - k1 (N2 - k1 for item 0, its own mirror)
      const float2 zm = a == 0 ? va[N2 - k1] : (b != a ? vb[N2 - 1 - k1] : va[N2 - 1 - k1]);
      if (b == a && 2 * k > H) continue;           // a self-mirrored item's upper half: done below
      // the pair (k0, h - k0), k0 <= h/2, as the separate split loop forms it
      const bool lo = 2 * k <= H;
      const int k0 = lo ? k : H - k;
      const float2 A = lo ? va[k1] : zm, Bc = lo ? zm : va[k1];
      const float2 E = make_float2(0.5f * (A.x + Bc.x), 0.5f * (A.y - Bc.y));
      const float2 D = make_float2(A.x - Bc.x, A.y + Bc.y);
      const float2 O = make_float2(0.5f * D.y, -0.5f * D.x);
      const float2 tt = cmul(twh[k0], O);
      const float2 xk = cadd(E, tt);
      X[k0] = make_float2(scale * xk.x, scale * xk.y);
      if (2 * k0 != H) {
        const float2 m = csub(E, tt);
        X[H - k0] = make_float2(scale * m.x, -scale * m.y);
      }
    }
  }
  __syncthreads();
}

// nr rows of half spectra staged in Xs (shared, pitch h + 1) to scaled real rows in g (Xs
// itself, or global memory; same pitch); the merge step as k_x_c2r (kernels.cu).  Z: rpc * PITCH.
// Ends with a barrier.
template <int N1, int N2>
__device__ __forceinline__ void xc2r4_staged(const float2* Xs, float2* g, int nr, float scale, const float2* tw,
                                             const float2* twh, float2* Z) {
  using L = RowLayout<N1, N2>;
  constexpr int H = L::H, PITCH = L::PITCH;
  constexpr int CN = H + 1;
  const int T = blockDim.x, tid = threadIdx.x;
  // pass 1 reads the half-length sequence z straight from the staged half spectrum: the merge
  // z[k] = (X[k] + conj X[h-k]) + i w^k (X[k] - conj X[h-k]) (w = e^{2 pi i / nxp}) computed
  // where pass 1 loads it, each z[k] with the operations of its pair's lower index k0 <= h/2
  // (z[h - k0] is the mirrored combination of the same terms)
  for (int q = tid; q < nr * N2; q += T) {
    const int r = q / N2, t = q - r * N2;
    const float2* X = Xs + r * CN;
    float2* z = Z + r * PITCH;
    four_step_pass1<N1, N2, 1>(
        t, tw,
        [&](int, int m) {
          const int k = t + N2 * m;
          if (k == 0) {
            const float a = X[0].x, b = X[H].x;
            return make_float2(a + b, a - b);
          }
          const bool lo = 2 * k <= H;
          const int k0 = lo ? k : H - k;
          const float2 xk = X[k0], xm = X[H - k0];
          const float2 P = make_float2(xk.x + xm.x, xk.y - xm.y);
          const float2 M = make_float2(xk.x - xm.x, xk.y + xm.y);
          const float2 w = twh[k0];
          const float2 Q = make_float2(M.x * w.x + M.y * w.y, M.y * w.x - M.x * w.y);
          return lo ? make_float2(P.x - Q.y, P.y + Q.x) : make_float2(P.x + Q.y, -P.y + Q.x);
        },
        [&](int, int k2, float2 v) { z[L::pad(t, k2)] = v; });
  }
  __syncthreads();
  for (int q = tid; q < nr * N1; q += T) {
    const int r = q / N1, k2 = q - r * N1;
    const float2* z = Z + r * PITCH;
    float2 v[N2];
    four_step_pass2<N1, N2, 1>(k2, [&](int k, int t) { return z[L::pad(t, k)]; }, v);
    float2* X = g + (size_t)r * CN;
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) {
      const float2 o = make_float2(v[k1].x * scale, v[k1].y * scale);
      X[k2 + N1 * k1] = o;
    }
    if (k2 == 0) X[H] = make_float2(0.f, 0.f);
  }
  __syncthreads();
}

// ------------------------------------------------------------------ inverse rows in pairs
//
// The inverse row transform of two rows at once (C2, fft_pair.cuh: the merge, both DFTs and the twiddles
// as packed instructions, one table read for both rows, the exchange between the passes in 16-byte words):
// 101 -> about 50 instructions a point at h = 270, where the scalar form ran at 60 % of the
// issue slots (540x540x256, 21 grids: 2.94 -> 2.47 ms, 78 % of the copy bandwidth; 768x768x320: 3.31
// -> 3.02).  One buffer serves the staged rows, the exchange words and the real rows: a thread
// has at most one item per pass, so all reads of a pass are over at the barrier before its writes.
// Lengths with N1 <= 24 (4 N1 registers of data); longer factors keep xc2r4_staged.
//
// B: the rows, pitch h + 1, pair p = rows 2 p, 2 p + 1; word (t, k2) of a pair's exchange buffer at
// t + k2 WS, an odd stride.  T >= ceil(nr / 2) max(N1, N2).  The real rows are left in B (the caller
// synchronises).
template <int N1, int N2>
struct RowPairs {
  static constexpr bool ok = N1 <= 24;
  static constexpr int H = N1 * N2, CN = H + 1, WS = N2 + (N2 % 2 == 0), PITCH = N1 * WS;
  // float2 of the buffer of np pairs
  static constexpr int words(int np) { return np * (2 * PITCH > 2 * CN ? 2 * PITCH : 2 * CN); }
};
template <int N1, int N2>
__device__ __forceinline__ void xc2r4_pairs(float2* B, int nr, float scale, const float2* tw, const float2* twh) {
  using L = RowPairs<N1, N2>;
  constexpr int H = L::H, CN = L::CN;
  const int np = (nr + 1) >> 1, tid = threadIdx.x;
  const uint32_t zb = smem_addr(B);
  C2 v[N1];
  const bool on1 = tid < np * N2;
  const int p1 = tid / N2, t = tid - p1 * N2;
  if (on1) {
    const float2* X0 = B + 2 * p1 * CN;
    const float2* X1 = 2 * p1 + 1 < nr ? X0 + CN : X0;
#pragma unroll
    for (int m = 0; m < N1; m++) {
      // z[k] = (X[k] + conj X[h-k]) + i w^k (X[k] - conj X[h-k]), w = e^{2 pi i / nxp}; a real-output
      // inverse has no slot for Im X[0], Im X[h]
      const int k = t + N2 * m;
      float2 a0 = X0[k], b0 = X0[H - k], a1 = X1[k], b1 = X1[H - k];
      if (m == 0 && t == 0) a0.y = b0.y = a1.y = b1.y = 0.f;
      const float2 w = twh[k];
      const float2 ar = make_float2(a0.x, a1.x), ai = make_float2(a0.y, a1.y);
      const float2 br = make_float2(b0.x, b1.x), bi = make_float2(b0.y, b1.y);
      const float2 pr = f2_add(ar, br), pi = f2_sub(ai, bi), mr = f2_sub(ar, br), mi = f2_add(ai, bi);
      const float2 qr = f2_fma(mi, f2_dup(w.y), f2_mul(mr, f2_dup(w.x)));
      const float2 qi = f2_fma(mr, f2_dup(-w.y), f2_mul(mi, f2_dup(w.x)));
      v[m] = {f2_sub(pr, qi), f2_add(pi, qr)};
    }
    DftP<N1, 1>::run(v);
#pragma unroll
    for (int k2 = 1; k2 < N1; k2++) {
      const float2 w = tw[t * k2];
      v[k2] = c2_mul(v[k2], w.x, -w.y);
    }
  }
  __syncthreads();
  if (on1) {
#pragma unroll
    for (int k2 = 0; k2 < N1; k2++) sts_c2(zb + 16u * (uint32_t)(p1 * L::PITCH + t + k2 * L::WS), v[k2]);
  }
  __syncthreads();
  const bool on2 = tid < np * N1;
  const int p2 = tid / N1, k2 = tid - p2 * N1;
  C2 u[N2];
  if (on2) {
#pragma unroll
    for (int t2 = 0; t2 < N2; t2++) u[t2] = lds_c2(zb + 16u * (uint32_t)(p2 * L::PITCH + t2 + k2 * L::WS));
    DftP<N2, 1>::run(u);
  }
  __syncthreads();
  if (on2) {
    float2* R0 = B + 2 * p2 * CN;
    const bool two = 2 * p2 + 1 < nr;
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) {
      const float2 r = f2_mul(u[k1].r, f2_dup(scale)), i = f2_mul(u[k1].i, f2_dup(scale));
      R0[k2 + N1 * k1] = make_float2(r.x, i.x);
      if (two) R0[CN + k2 + N1 * k1] = make_float2(r.y, i.y);
    }
    if (k2 == 0) {
      R0[H] = make_float2(0.f, 0.f);
      if (two) R0[CN + H] = make_float2(0.f, 0.f);
    }
  }
}

// L2 prefetch of the row chunk pf block indices on (x fastest): rows of (h + 1) complex values,
// chunks of rpc rows, blockIdx.y the grid; from gs.src (FWD) or gs.p.
template <bool FWD>
__device__ __forceinline__ void x4_prefetch(const GridSet& gs, int rows, int rpc, int CN, int pf) {
  const int tn = blockIdx.y * gridDim.x + blockIdx.x + pf;
  if (threadIdx.x != 0 || tn >= (int)(gridDim.x * gridDim.y)) return;
  const int gy = tn / gridDim.x, c = tn - gy * gridDim.x;
  const int row0 = c * rpc, nr = min(rpc, rows - row0);
  const float2* s = reinterpret_cast<const float2*>(FWD ? gs.src[gy] : gs.p[gy]) + (size_t)row0 * CN;
  const size_t n = (size_t)nr * CN;
  // in pieces of 64 KB
  for (size_t o = 0; o < n; o += 8192) l2_prefetch(s + o, 8u * min((size_t)8192, n - o), s, s + n);
}

// ------------------------------------------------------------------ staged row chunks
//
// A chunk of rows is one contiguous run of global memory.  It comes in by 16-byte cp.async and
// its results, written over it in shared memory, leave by one bulk copy (cp.async.bulk, issued by
// one thread), so the passes spend no instructions on global addresses and every global access is
// a full line.  al: 16 where the chunk starts on a 16-byte boundary (the grid is 16-byte aligned and the
// chunk starts at an even row: two rows are a multiple of 16 bytes whatever nxp is); 8 otherwise: both
// ways move 8-byte words; 4 where the real input of an odd length starts off an 8-byte boundary, which needs
// no more than a float's alignment (its rows were never read as pairs): 4-byte words in.

// n 8-byte words from src to dst (shared, 16-byte aligned); the caller commits and waits.
__device__ __forceinline__ void rows_in(float2* dst, const float2* src, int n, int al) {
  const uint32_t d = smem_addr(dst);
  if (al == 16) {
    const int n2 = n >> 1;
    for (int e = threadIdx.x; e < n2; e += blockDim.x) cp_async16(d + 16u * (uint32_t)e, src + 2 * e);
    if ((n & 1) && threadIdx.x == 0) cp_async8(d + 8u * (uint32_t)(n - 1), src + n - 1);
  } else if (al == 8) {
    for (int e = threadIdx.x; e < n; e += blockDim.x) cp_async8(d + 8u * (uint32_t)e, src + e);
  } else {
    const float* f = reinterpret_cast<const float*>(src);
    for (int e = threadIdx.x; e < 2 * n; e += blockDim.x) cp_async4(d + 4u * (uint32_t)e, f + e);
  }
  cp_async_commit();
}

// n 8-byte words from src (shared, 16-byte aligned, written by this CTA's threads, no barrier
// since) to dst.  Returns when shared memory may be given back.
__device__ __forceinline__ void rows_out(float2* dst, const float2* src, int n, int al) {
  if (al == 16) {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t bytes = 8u * (uint32_t)(n & ~1);
      if (bytes)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(
                         __cvta_generic_to_global(dst)),
                     "r"(smem_addr(src)), "r"(bytes)
                     : "memory");
      asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      if (n & 1) dst[n - 1] = src[n - 1];
      asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
    }
  } else {
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) dst[e] = src[e];
  }
}

// The forward rows keep their loads and stores in the passes: pass 1's loads are the first thing a
// thread does and pass 2 stores runs of N1 points; staged both ways they measured slower (540x540x256:
// 1.24 against 1.18 ms; staged stores alone the same), the rows' second buffer costing resident CTAs.
//
// the counters a job clears with its first transform
__device__ __forceinline__ void x_clear(const GridSet& gs) {
  if (gs.zero && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < kNumCounters) gs.zero[threadIdx.x] = 0;
}

// stage != 0: the twiddle tables are copied into shared memory first; 0: the passes read
// them from global memory (L1-resident: every CTA of the launch reads the same 2 h values),
// and the CTA's first barrier and the table copy go away.
template <int N1, int N2>
__global__ void __launch_bounds__(256) k_xr2c4(const __grid_constant__ GridSet gs, int rows, int rpc,
                                               const float2* __restrict__ twg, const float2* __restrict__ twn,
                                               int stage, int pf) {
  constexpr int H = N1 * N2;
  extern __shared__ float2 sm[];
  const float2 *tw = twg, *twh = twn;
  float2* Z = sm;
  dep_wait();
  dep_launch();
  x_clear(gs);
  if (pf > 0) x4_prefetch<true>(gs, rows, rpc, H + 1, pf);
  if (stage) {
    float2* t1 = sm;
    float2* t2 = t1 + H;
    for (int t = threadIdx.x; t < H; t += blockDim.x) {
      t1[t] = twg[t];
      t2[t] = twn[t];
    }
    tw = t1;
    twh = t2;
    Z = t2 + H;
    __syncthreads();
  }
  const int row0 = blockIdx.x * rpc, nr = min(rpc, rows - row0);
  const float2* src = reinterpret_cast<const float2*>(gs.src[blockIdx.y]) + (size_t)row0 * (H + 1);
  float2* dst = reinterpret_cast<float2*>(gs.p[blockIdx.y]) + (size_t)row0 * (H + 1);
  xr2c4_rows<N1, N2>(src, dst, nr, gs.scale[blockIdx.y], tw, twh, Z);
}

template <int N1, int N2>
__global__ void __launch_bounds__(256) k_xc2r4(const __grid_constant__ GridSet gs, int rows, int rpc,
                                               const float2* __restrict__ twg, const float2* __restrict__ twn,
                                               int al, int pf) {
  constexpr int H = N1 * N2, CN = H + 1;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  float2* twh = tw + H;
  float2* Xs = sm + 2 * H;
  const int row0 = blockIdx.x * rpc, nr = min(rpc, rows - row0);
  float2* g = reinterpret_cast<float2*>(gs.p[blockIdx.y]) + (size_t)row0 * CN;
  dep_wait();
  dep_launch();
  rows_in(Xs, g, nr * CN, al);
  if (pf > 0) x4_prefetch<false>(gs, rows, rpc, CN, pf);
  for (int t = threadIdx.x; t < H; t += blockDim.x) {
    tw[t] = twg[t];
    twh[t] = twn[t];
  }
  cp_async_wait_0();
  __syncthreads();
  if constexpr (RowPairs<N1, N2>::ok) xc2r4_pairs<N1, N2>(Xs, nr, gs.scale[blockIdx.y], tw, twh);
  else xc2r4_staged<N1, N2>(Xs, Xs, nr, gs.scale[blockIdx.y], tw, twh, Xs + even_up(rpc * CN));
  rows_out(g, Xs, nr * CN, al);
}

// ------------------------------------------------------------------ rows, odd nxp
//
// Odd lengths N = N1 N2 have no half-length form: two rows a, b go through one complex transform
// of z = a + i b, so a row costs what half a complex line costs, as in the even form.
//   forward  A[k] = (Z[k] + conj Z[N-k]) / 2,  B[k] = (Z[k] - conj Z[N-k]) / 2i;
//            item k2 and its mirror N1 - k2 of pass 2 sit in one thread, which then holds Z[k] and
//            Z[N-k] for all its k (as xr2c4_rows)
//   inverse  Z[k] = A[k] + i B[k] (k <= N/2), Z[N-k] = conj A[k] + i conj B[k], formed where pass 1
//            loads it; Im A[0] and Im B[0] have no slot in a real-output transform
// A row so carries the rounding of the larger of its pair: a zero row beside a large one comes back as some 1e-7 of
// that one, as the y and z transforms leave every line within 1e-7 of its largest point.
// Rows in global and staged memory have N + 1 floats; the last is written as zero.
template <int N1, int N2>
__global__ void __launch_bounds__(256) k_xr2c4o(const __grid_constant__ GridSet gs, int rows, int lpc,
                                                const float2* __restrict__ twg, int al) {
  using L = RowLayout<N1, N2>;
  constexpr int N = N1 * N2, CN = (N + 1) / 2, NPI = N1 / 2 + 1;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  float2* Xs = sm + even_up(N);
  float2* Z = Xs + 2 * lpc * CN;
  const int T = blockDim.x, tid = threadIdx.x;
  const int row0 = blockIdx.x * 2 * lpc, nr = min(2 * lpc, rows - row0), nl = (nr + 1) / 2;
  const size_t o = (size_t)row0 * CN;
  dep_wait();
  dep_launch();
  x_clear(gs);
  rows_in(Xs, reinterpret_cast<const float2*>(gs.src[blockIdx.y]) + o, nr * CN, al);
  for (int t = tid; t < N; t += T) tw[t] = twg[t];
  cp_async_wait_0();
  __syncthreads();
  const float* Xf = reinterpret_cast<const float*>(Xs);
  for (int q = tid; q < nl * N2; q += T) {
    const int l = q / N2, t = q - l * N2;
    const float* a = Xf + 2 * l * (N + 1) + t;
    const bool two = 2 * l + 1 < nr;
    float2* z = Z + l * L::PITCH;
    four_step_pass1<N1, N2, -1>(
        t, tw, [&](int, int m) { return make_float2(a[m * N2], two ? a[N + 1 + m * N2] : 0.f); },
        [&](int, int k2, float2 v) { z[L::pad(t, k2)] = v; });
  }
  __syncthreads();
  const float hs = 0.5f * gs.scale[blockIdx.y];
  for (int q = tid; q < nl * NPI; q += T) {
    const int l = q / NPI, a = q - l * NPI;
    const float2* z = Z + l * L::PITCH;
    float2 va[N2], vb[N2];
    four_step_pass2<N1, N2, -1>(a, [&](int k, int t) { return z[L::pad(t, k)]; }, va);
    if (a != 0) four_step_pass2<N1, N2, -1>(N1 - a, [&](int k, int t) { return z[L::pad(t, k)]; }, vb);
    float2* XA = Xs + 2 * l * CN;
    const bool two = 2 * l + 1 < nr;
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) {
      const int k = a + N1 * k1;
      if (k == 0) {
        XA[0] = make_float2(2.f * hs * va[0].x, 0.f);
        if (two) XA[CN] = make_float2(2.f * hs * va[0].y, 0.f);
        continue;
      }
      if (a == 0 && 2 * k > N) continue;     // item 0 mirrors itself: its upper half is done below
      const float2 zm = a == 0 ? va[N2 - k1] : vb[N2 - 1 - k1];
      const bool lo = 2 * k < N;
      const int k0 = lo ? k : N - k;
      const float2 p = lo ? va[k1] : zm, m = lo ? zm : va[k1];   // Z[k0], Z[N - k0]
      XA[k0] = make_float2(hs * (p.x + m.x), hs * (p.y - m.y));
      if (two) XA[CN + k0] = make_float2(hs * (p.y + m.y), hs * (m.x - p.x));
    }
  }
  rows_out(reinterpret_cast<float2*>(gs.p[blockIdx.y]) + o, Xs, nr * CN, al);
}

template <int N1, int N2>
__global__ void __launch_bounds__(256) k_xc2r4o(const __grid_constant__ GridSet gs, int rows, int lpc,
                                                const float2* __restrict__ twg, int al) {
  using L = RowLayout<N1, N2>;
  constexpr int N = N1 * N2, CN = (N + 1) / 2;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  float2* Xs = sm + even_up(N);
  float2* Z = Xs + 2 * lpc * CN;
  const int T = blockDim.x, tid = threadIdx.x;
  const int row0 = blockIdx.x * 2 * lpc, nr = min(2 * lpc, rows - row0), nl = (nr + 1) / 2;
  float2* g = reinterpret_cast<float2*>(gs.p[blockIdx.y]) + (size_t)row0 * CN;
  dep_wait();
  dep_launch();
  rows_in(Xs, g, nr * CN, al);
  for (int t = tid; t < N; t += T) tw[t] = twg[t];
  cp_async_wait_0();
  __syncthreads();
  for (int q = tid; q < nl * N2; q += T) {
    const int l = q / N2, t = q - l * N2;
    const float2* XA = Xs + 2 * l * CN;
    const bool two = 2 * l + 1 < nr;
    float2* z = Z + l * L::PITCH;
    four_step_pass1<N1, N2, 1>(
        t, tw,
        [&](int, int m) {
          const int k = t + N2 * m;
          const bool lo = 2 * k < N;
          const int k0 = lo ? k : N - k;
          float2 a = XA[k0], b = two ? XA[CN + k0] : make_float2(0.f, 0.f);
          if (k == 0) a.y = b.y = 0.f;
          return lo ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, b.x - a.y);
        },
        [&](int, int k2, float2 v) { z[L::pad(t, k2)] = v; });
  }
  __syncthreads();
  const float scale = gs.scale[blockIdx.y];
  float* Xf = reinterpret_cast<float*>(Xs);
  for (int q = tid; q < nl * N1; q += T) {
    const int l = q / N1, k2 = q - l * N1;
    const float2* z = Z + l * L::PITCH;
    float2 v[N2];
    four_step_pass2<N1, N2, 1>(k2, [&](int k, int t) { return z[L::pad(t, k)]; }, v);
    float* a = Xf + 2 * l * (N + 1);
    const bool two = 2 * l + 1 < nr;
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) {
      a[k2 + N1 * k1] = v[k1].x * scale;
      if (two) a[N + 1 + k2 + N1 * k1] = v[k1].y * scale;
    }
    if (k2 == 0) {
      a[N] = 0.f;
      if (two) a[2 * N + 1] = 0.f;
    }
  }
  rows_out(g, Xs, nr * CN, al);
}

static inline cudaError_t resident_grid(const void* fn, int T, size_t smem, int units, int* grid) {
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, T, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  *grid = std::max(1, std::min(units, per_sm * nsm));
  return cudaSuccess;
}

// ------------------------------------------------------------------ launch templates

static inline bool four_step_enabled(int n) { return tuned("four_step", n, 1) != 0; }

static inline int round_up32(int t) { return std::max(64, (t + 31) / 32 * 32); }

template <int N1, int N2, int DIR>
static cudaError_t line4_scalar(const GridSet& gs, int ni, size_t pstride, int no, size_t ostride, const float2* tw,
                         cudaStream_t st) {
  constexpr int N = N1 * N2;
  // 8-column tiles; 16 for inverse transforms up to 540 points (measured faster there,
  // slower at 768)
  int W = std::max(1, tuned(DIR < 0 ? "line4_w_fwd" : "line4_w_inv", N, (DIR > 0 && N <= 540) ? 16 : 8));
  while (W > 1 && W / 2 >= ni) W /= 2;
  int lw = 0;
  while ((1 << lw) < W) lw++;
  W = 1 << lw;
  const int SK = W < 16 ? (((W - N2 * W) % 16) + 16) % 16 : 0;
  // threads per CTA: by default one item per thread of the longer pass up to 256; the
  // schedule may set up to 512 (a whole number of warps), e.g. so that one pass runs in a
  // single round
  int T = std::min(256, round_up32(W * std::max(N1, N2)));
  T = std::max(64, std::min(DIR < 0 ? 256 : 512,
                            tuned(DIR < 0 ? "line4_threads_fwd" : "line4_threads_inv", N, T) / 32 * 32));
  const int nIT = (ni + W - 1) / W;
  const size_t smem = sizeof(float2) * (size_t)N + line4_smem<N1, N2>(W, SK);
  const auto fn = k_line4s<N1, N2, DIR>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)(nIT * no), gs.n);
  // L2 line prefetch ahead of the tiles: schedule keys line4_pf_fwd / line4_pf_inv, the distance in
  // quarters of the resident tiles (0 = off)
  int pf = 0;
  if (const int q = tuned(DIR < 0 ? "line4_pf_fwd" : "line4_pf_inv", N, 0)) {
    int res = 0;
    if ((e = resident_grid((const void*)fn, T, smem, 1 << 30, &res)) != cudaSuccess) return e;
    pf = std::max(1, res * q / 4);
  }
  const size_t bytes = sizeof(float2) * (size_t)gs.n * ni * N * no;
  return launch_dep(bytes, fn, grid, T, smem, st, gs, ni, pstride, ostride, W, lw, nIT, SK, tw, pf);
}

template <int N, int DIR>
static cudaError_t line4_pairs(const GridSet& gs, int ni, size_t pstride, int no, size_t ostride, const float2* tw,
                               cudaStream_t st) {
  constexpr ColSplit S = col_split(N);
  // 16-column tiles (rows of 128 bytes); narrower where the grid is
  int W = std::max(2, std::min(16, tuned(DIR < 0 ? "line4_w_fwd" : "line4_w_inv", N, 16)));
  while (W > 2 && W / 2 >= ni) W /= 2;
  int lnp = 0;
  while ((4 << lnp) <= W) lnp++;
  W = 2 << lnp;
  const size_t smem = sizeof(float2) * ((size_t)even_up(N) + (size_t)W * N);
  // threads: the items of the first stage in as few rounds of at most 256 threads as they take
  const int items = (W / 2) * (N / S.r0), rounds = (items + 255) / 256;
  int T = round_up32((items + rounds - 1) / rounds);
  // one warp more where it saves both other stages a round (252 = 7 x 6 x 6: 160 threads 176 us, 192 135, inverse, 21 grids)
  if constexpr (S.r2 > 1) {
    const int i1 = (W / 2) * (N / S.r1), i2 = (W / 2) * (N / S.r2), up = T + 32;
    if (up <= 256 && (i1 - 1) / up < (i1 - 1) / T && (i2 - 1) / up < (i2 - 1) / T) T = up;
  }
  T = std::max(64, std::min(256, tuned(DIR < 0 ? "line4_threads_fwd" : "line4_threads_inv", N, T) / 32 * 32));
  const int nIT = (ni + W - 1) / W;
  const auto fn = k_line4<N, DIR>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)(nIT * no), gs.n);
  const size_t bytes = sizeof(float2) * (size_t)gs.n * ni * N * no;
  return launch_dep(bytes, fn, grid, T, smem, st, gs, ni, pstride, ostride, lnp, nIT, tw);
}

// Which columns of up to 270 points go in pairs (above, three stages cost more than the scalar form's two); time of the
// scalar form over the pairs', y columns of jobs with 21 grids of 250 x-points, and z lines of one 540x540 plane set:
//   scalar split with a factor above 20   1.33-1.92 (125, 147, 175, 189, 243, 250 points), z lines 1.12-1.54
//   up to 180 points                      1.00-1.23, z lines 0.99-1.09
//   above, forward                        1.00-1.13 (252 points 0.96), z lines 0.99-1.16
//   above, inverse                        0.91-1.03, z lines 0.96-1.01, but 1.04-1.13 with 64 x-points: there the
//                                         scalar form, its tiles too few to hide its longer rounds, is the slower
template <int N1, int N2>
static cudaError_t line4(const GridSet& gs, int ni, size_t pstride, int no, size_t ostride, const float2* tw,
                         float sign, cudaStream_t st) {
  constexpr int N = N1 * N2;
  if constexpr (N <= 270) {
    if (sign > 0.f && (N1 > 20 || N <= 180 || ni <= 64)) return line4_pairs<N, 1>(gs, ni, pstride, no, ostride, tw, st);
    // residual spectra keep the scalar form's order of roundings in their forward transforms
    if (sign < 0.f && !gs.plain) return line4_pairs<N, -1>(gs, ni, pstride, no, ostride, tw, st);
  }
  return sign < 0.f ? line4_scalar<N1, N2, -1>(gs, ni, pstride, no, ostride, tw, st)
                    : line4_scalar<N1, N2, 1>(gs, ni, pstride, no, ostride, tw, st);
}

// Threads and lines per CTA of a row kernel whose passes have i1 and i2 items per line of c1 and
// c2 points each.  A CTA's time is its rounds of T items, each as long as its item, plus a fixed
// part; per line an SM spends that time over the lines it has in flight (latency), and the issue
// slots of the T threads, idle ones of a short pass included.  (125 = 25 x 5 at 64 threads and 2
// lines had 10 busy threads in pass 1: 250x250x200, 21 grids 1.93 ms, with this rule 0.52.)  At
// most 36 KB of shared memory, so that six CTAs share an SM; lines a multiple of step.
struct RowShape {
  int T, lines;
};
static inline RowShape row_shape(int i1, int c1, int i2, int c2, size_t fixed, size_t per_line, int step) {
  RowShape best{64, step};
  double least = 1e30;
  for (int T = 64; T <= 256; T += 32)
    for (int n = step; n <= 64; n += step) {
      const size_t smem = fixed + n * per_line + 1024;
      if (n > step && smem > 37 * 1024) break;
      const int ctas = std::min(32, std::min((int)(227 * 1024 / smem), 65536 / (96 * T)));
      const double d = (n * i1 + T - 1) / T * (4 + c1) + (n * i2 + T - 1) / T * (4 + c2) + 12;
      const double t = d / n * (40.0 / std::max(1, ctas) + 2.5 * T / 32);
      if (t < least * 0.999) {
        least = t;
        best = {T, n};
      }
    }
  return best;
}

// the alignment that every grid of the set has, inputs (of a forward transform) included: 16, 8 or 4
static inline int grids_align(const GridSet& gs, bool fwd) {
  uintptr_t a = 0;
  for (int q = 0; q < gs.n; q++) a |= reinterpret_cast<uintptr_t>(gs.p[q]) | (fwd ? reinterpret_cast<uintptr_t>(gs.src[q]) : 0);
  return a % 16 == 0 ? 16 : a % 8 == 0 ? 8 : 4;
}

// Row pairs per CTA of xc2r4_pairs: one item per thread and pass, by the same estimate as row_shape.
template <int N1, int N2>
static inline int pair_count() {
  using L = RowPairs<N1, N2>;
  int best = 1;
  double least = 1e30;
  for (int np = 1; np * N1 <= 256; np++) {
    const size_t smem = sizeof(float2) * (2 * (size_t)L::H + L::words(np)) + 1024;
    if (np > 1 && smem > 37 * 1024) break;
    const int T = std::max(64, (np * N1 + 31) / 32 * 32);
    const int ctas = std::min(32, std::min((int)(227 * 1024 / smem), 65536 / ((4 * N1 + 40) * T)));
    const double t = (40.0 / std::max(1, ctas) + 2.5 * T / 32) / np;
    if (t < least * 0.999) {
      least = t;
      best = np;
    }
  }
  return best;
}

template <int N1, int N2>
static cudaError_t x4(bool fwd, const GridSet& gs, int rows, const float2* tw, const float2* twn, cudaStream_t st) {
  using L = RowLayout<N1, N2>;
  constexpr int H = L::H;
  constexpr bool kPairs = RowPairs<N1, N2>::ok;
  // twiddle tables staged in shared memory (schedule key x4_stage_fwd) or read from global memory
  const int stage = !fwd || tuned("x4_stage_fwd", H, 1) != 0;
  const size_t fixed = sizeof(float2) * 2 * (size_t)H * stage;
  const size_t per = sizeof(float2) * (size_t)(L::PITCH + (fwd ? 0 : H + 1));
  // the forward form, whose loads go straight into pass 1, is faster at 128 threads with one item
  // pair each (270x270x256: 0.24 against 0.29 ms) unless that leaves half of pass 1 idle
  // (250x250x200: 0.25 against 0.19 ms)
  RowShape rs{128, 128 / (N1 / 2 + 1)};
  if (!fwd || rs.lines < 1 || 2 * rs.lines * N2 < rs.T)
    rs = row_shape(N2, N1, fwd ? N1 / 2 + 1 : N1, fwd ? 2 * N2 : N2, fixed, per, fwd ? 1 : 2);
  int rpc = std::max(1, std::min(64, tuned(fwd ? "x4_rpc_fwd" : "x4_rpc_inv", H, rs.lines)));
  int T = std::max(64, std::min(256, tuned(fwd ? "x4_threads_fwd" : "x4_threads_inv", H, rs.T) / 32 * 32));
  size_t smem = fixed + per * rpc + sizeof(float2);
  if constexpr (kPairs) {
    if (!fwd) {
      const int np = std::max(1, std::min(256 / N1, tuned("x4_rpc_inv", H, 2 * pair_count<N1, N2>()) / 2));
      rpc = 2 * np;
      T = std::max(64, std::max((np * N1 + 31) / 32 * 32, std::min(256, tuned("x4_threads_inv", H, 64) / 32 * 32)));
      smem = fixed + sizeof(float2) * RowPairs<N1, N2>::words(np);
    }
  }
  const void* fn = fwd ? (const void*)k_xr2c4<N1, N2> : (const void*)k_xc2r4<N1, N2>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((rows + rpc - 1) / rpc), gs.n);
  // L2 prefetch of the row chunk ahead of the CTAs (schedule keys x4_pf_fwd / x4_pf_inv: the
  // distance in quarters of the resident CTAs, 0 = off)
  int pf = 0;
  if (const int q = tuned(fwd ? "x4_pf_fwd" : "x4_pf_inv", H, fwd ? 4 : 0)) {
    int res = 0;
    if ((e = resident_grid(fn, T, smem, 1 << 30, &res)) != cudaSuccess) return e;
    pf = std::max(1, res * q / 4);
  }
  // every chunk starts at an even row, or two rows' bytes do not matter ((h + 1) even)
  const int al = std::min(grids_align(gs, fwd), rpc % 2 == 0 || (H + 1) % 2 == 0 ? 16 : 8);
  const size_t bytes = sizeof(float2) * (size_t)gs.n * rows * (H + 1);
  return fwd ? launch_dep(bytes, k_xr2c4<N1, N2>, grid, T, smem, st, gs, rows, rpc, tw, twn, stage, pf)
             : launch_dep(bytes, k_xc2r4<N1, N2>, grid, T, smem, st, gs, rows, rpc, tw, twn, al, pf);
}

// odd nxp = N1 N2: rows taken in pairs
template <int N1, int N2>
static cudaError_t x4_odd(bool fwd, const GridSet& gs, int rows, const float2* tw, cudaStream_t st) {
  using L = RowLayout<N1, N2>;
  constexpr int N = N1 * N2;
  const size_t fixed = sizeof(float2) * even_up(N), per = sizeof(float2) * (size_t)(L::PITCH + N + 1);
  const RowShape rs = row_shape(N2, N1, fwd ? N1 / 2 + 1 : N1, fwd ? 2 * N2 : N2, fixed, per, 1);
  const size_t smem = fixed + per * rs.lines;
  const void* fn = fwd ? (const void*)k_xr2c4o<N1, N2> : (const void*)k_xc2r4o<N1, N2>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((rows + 2 * rs.lines - 1) / (2 * rs.lines)), gs.n);
  const int al = grids_align(gs, fwd);
  const size_t bytes = sizeof(float) * (size_t)gs.n * rows * (N + 1);
  return fwd ? launch_dep(bytes, k_xr2c4o<N1, N2>, grid, rs.T, smem, st, gs, rows, rs.lines, tw, al)
             : launch_dep(bytes, k_xc2r4o<N1, N2>, grid, rs.T, smem, st, gs, rows, rs.lines, tw, al);
}

}  // namespace crava

// Register DFTs on pairs of complex values (sm_100a).
//
// A C2 holds the same point of two independent lines, real parts in one float2 and imaginary
// parts in the other, so that every addition, multiplication and twiddle of a transform is one
// packed instruction (add / sub / mul / fma .rn.f32x2) for both lines.  The packed forms run at
// the scalar forms' flop rate (measured: 2 packed against 4 scalar warp instructions per clock and
// SM), but take half the issue slots; the transforms in the pencil pass are bound by issue and
// latency, not by the FP32 pipe.  Each half is rounded like the scalar operation.
#pragma once
#include "fft2.cuh"

namespace crava {

__device__ __forceinline__ unsigned long long f2_bits(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 f2_from(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_from(r);
}
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_from(r);
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_from(r);
}
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
  return f2_from(r);
}
__device__ __forceinline__ float2 f2_dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2_neg(float2 a) { return make_float2(-a.x, -a.y); }

struct C2 {
  float2 r, i;
};
__device__ __forceinline__ C2 c2_add(C2 a, C2 b) { return {f2_add(a.r, b.r), f2_add(a.i, b.i)}; }
__device__ __forceinline__ C2 c2_sub(C2 a, C2 b) { return {f2_sub(a.r, b.r), f2_sub(a.i, b.i)}; }
// a + S i b
template <int S>
__device__ __forceinline__ C2 c2_add_i(C2 a, C2 b) {
  return S > 0 ? C2{f2_sub(a.r, b.i), f2_add(a.i, b.r)} : C2{f2_add(a.r, b.i), f2_sub(a.i, b.r)};
}
// a + c b (c real)
__device__ __forceinline__ C2 c2_fma(float c, C2 b, C2 a) {
  return {f2_fma(f2_dup(c), b.r, a.r), f2_fma(f2_dup(c), b.i, a.i)};
}
__device__ __forceinline__ C2 c2_scale(C2 a, float c) { return {f2_mul(a.r, f2_dup(c)), f2_mul(a.i, f2_dup(c))}; }
// a (wr + i wi), both lines by the same factor
__device__ __forceinline__ C2 c2_mul(C2 a, float wr, float wi) {
  const float2 x = f2_dup(wr), y = f2_dup(wi);
  return {f2_fma(a.i, f2_dup(-wi), f2_mul(a.r, x)), f2_fma(a.r, y, f2_mul(a.i, x))};
}
// a e^{S 2 pi i m / R}, m and R constants after unrolling: multiples of an eighth turn by
// additions
template <int S, int R>
__device__ __forceinline__ C2 c2_turn(C2 a, int m) {
  m = ((S * m) % R + R) % R;
  constexpr float h = SQRT1_2;
  if ((8 * m) % R == 0) {
    switch (8 * m / R) {
      case 0: return a;
      case 1: return {f2_mul(f2_sub(a.r, a.i), f2_dup(h)), f2_mul(f2_add(a.i, a.r), f2_dup(h))};
      case 2: return {f2_neg(a.i), a.r};
      case 3: return {f2_mul(f2_add(a.r, a.i), f2_dup(-h)), f2_mul(f2_sub(a.r, a.i), f2_dup(h))};
      case 4: return {f2_neg(a.r), f2_neg(a.i)};
      case 5: return {f2_mul(f2_sub(a.i, a.r), f2_dup(h)), f2_mul(f2_add(a.r, a.i), f2_dup(-h))};
      case 6: return {a.i, f2_neg(a.r)};
      default: return {f2_mul(f2_add(a.r, a.i), f2_dup(h)), f2_mul(f2_sub(a.i, a.r), f2_dup(h))};
    }
  }
  return c2_mul(a, TwG<R>::c(m), TwG<R>::s(m));
}

// y_m = sum_r v_r e^{S 2 pi i r m / R} of both lines, in place
template <int R, int S>
struct DftP {
  static __device__ __forceinline__ void run(C2* v) {
    constexpr int A = codelet_split(R), B = R / A;
    C2 u[A][B];
#pragma unroll
    for (int r1 = 0; r1 < A; r1++) {
#pragma unroll
      for (int r2 = 0; r2 < B; r2++) u[r1][r2] = v[r1 + A * r2];
      DftP<B, S>::run(u[r1]);
      if (r1 > 0) {
#pragma unroll
        for (int k2 = 1; k2 < B; k2++) u[r1][k2] = c2_turn<S, R>(u[r1][k2], r1 * k2);
      }
    }
#pragma unroll
    for (int k2 = 0; k2 < B; k2++) {
      C2 t[A];
#pragma unroll
      for (int r1 = 0; r1 < A; r1++) t[r1] = u[r1][k2];
      DftP<A, S>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) v[k2 + B * k1] = t[k1];
    }
  }
};

template <int S>
struct DftP<2, S> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 a = v[0], b = v[1];
    v[0] = c2_add(a, b);
    v[1] = c2_sub(a, b);
  }
};
template <int S>
struct DftP<3, S> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 t1 = c2_add(v[1], v[2]), t2 = c2_scale(c2_sub(v[1], v[2]), C3_S);
    const C2 m = c2_fma(-0.5f, t1, v[0]);
    v[0] = c2_add(v[0], t1);
    v[1] = c2_add_i<S>(m, t2);
    v[2] = c2_add_i<-S>(m, t2);
  }
};
template <int S>
struct DftP<4, S> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 a = c2_add(v[0], v[2]), b = c2_sub(v[0], v[2]);
    const C2 c = c2_add(v[1], v[3]), d = c2_sub(v[1], v[3]);
    v[0] = c2_add(a, c);
    v[2] = c2_sub(a, c);
    v[1] = c2_add_i<S>(b, d);
    v[3] = c2_add_i<-S>(b, d);
  }
};
template <int S>
struct DftP<5, S> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 a1 = c2_add(v[1], v[4]), b1 = c2_sub(v[1], v[4]);
    const C2 a2 = c2_add(v[2], v[3]), b2 = c2_sub(v[2], v[3]);
    const C2 c1 = c2_fma(C5_C2, a2, c2_fma(C5_C1, a1, v[0]));
    const C2 c2 = c2_fma(C5_C1, a2, c2_fma(C5_C2, a1, v[0]));
    const C2 s1 = c2_fma(C5_S2, b2, c2_scale(b1, C5_S1));
    const C2 s2 = c2_fma(-C5_S1, b2, c2_scale(b1, C5_S2));
    v[0] = c2_add(c2_add(v[0], a1), a2);
    v[1] = c2_add_i<S>(c1, s1);
    v[4] = c2_add_i<-S>(c1, s1);
    v[2] = c2_add_i<S>(c2, s2);
    v[3] = c2_add_i<-S>(c2, s2);
  }
};
template <int S>
struct DftP<7, S> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 a1 = c2_add(v[1], v[6]), b1 = c2_sub(v[1], v[6]);
    const C2 a2 = c2_add(v[2], v[5]), b2 = c2_sub(v[2], v[5]);
    const C2 a3 = c2_add(v[3], v[4]), b3 = c2_sub(v[3], v[4]);
    const C2 c1 = c2_fma(C7_C3, a3, c2_fma(C7_C2, a2, c2_fma(C7_C1, a1, v[0])));
    const C2 c2 = c2_fma(C7_C1, a3, c2_fma(C7_C3, a2, c2_fma(C7_C2, a1, v[0])));
    const C2 c3 = c2_fma(C7_C2, a3, c2_fma(C7_C1, a2, c2_fma(C7_C3, a1, v[0])));
    const C2 s1 = c2_fma(C7_S3, b3, c2_fma(C7_S2, b2, c2_scale(b1, C7_S1)));
    const C2 s2 = c2_fma(-C7_S1, b3, c2_fma(-C7_S3, b2, c2_scale(b1, C7_S2)));
    const C2 s3 = c2_fma(C7_S2, b3, c2_fma(-C7_S1, b2, c2_scale(b1, C7_S3)));
    v[0] = c2_add(c2_add(c2_add(v[0], a1), a2), a3);
    v[1] = c2_add_i<S>(c1, s1);
    v[6] = c2_add_i<-S>(c1, s1);
    v[2] = c2_add_i<S>(c2, s2);
    v[5] = c2_add_i<-S>(c2, s2);
    v[3] = c2_add_i<S>(c3, s3);
    v[4] = c2_add_i<-S>(c3, s3);
  }
};

// four floats of shared memory at byte address a
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ C2 lds_c2(uint32_t a) {
  const float4 v = lds4(a);
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void sts_c2(uint32_t a, C2 v) { sts4(a, make_float4(v.r.x, v.r.y, v.i.x, v.i.y)); }

}  // namespace crava

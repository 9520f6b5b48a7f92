// Classical (far) limit of a primitive quartet: for rho |PQ|^2 above a bound
// the Boys function is its asymptote, F_m(T) = (2m-1)!! / (2T)^m F_0(T) with
// F_0 = sqrt(pi / T) / 2, and every factor sqrt(1/(p+q)) or rho of the
// Obara-Saika recursion cancels: a step of the recursion that raises m by one
// carries exactly one factor rho (W-P = -rho/p PQ, -rho/p, rho/(2pq)), and
// rho^m F_m / sqrt(rho) depends on |PQ| alone.  With
//   I_m = k_ab k_cd (2m-1)!! / (2^m R^{2m+1}),  k = K sqrt(sqrt(pi)/2) / sqrt(p),
//   WP = -PQ/p,  WQ = PQ/q,  nrp = -1/p,  nrq = -1/q,  o2pq = 1/(2pq)
// the generated recursions give the same integrals from one reciprocal
// square root: no 1/sqrt(p+q), no Boys table row, no exponential.
#pragma once
#include <cuda_runtime.h>

#include "quartet.cuh"

namespace pyfacc {

using ::pf_fma;  // the scalar forms, beside F2's

// Lower bound on T = rho |PQ|^2 of a far quartet of total angular momentum L.
// The neglected part of F_m relative to F_m is Gamma(m+1/2, T) / Gamma(m+1/2):
// below 3e-16 for m <= L at 36 + 3L in FP64, below 3e-8 at 17 + 3L in FP32.
template <typename R> __host__ __device__ constexpr float far_tmin(int L) {
  return sizeof(R) == 8 ? 36.0f + 3.0f * L : 17.0f + 3.0f * L;
}

// Whether every primitive quartet of two shell pairs is far:
// |PQ| >= sqrt(tmin (s_i + s_j)) with s = 1/p, 1/q for all i, j.  With
// sqrt(s_i + s_j) <= (s_i + s_j) / (2c) + c/2 (the tangent at s_i + s_j = c^2)
// and |PQ| >= |CC'| - r_i - r_j (r: distance of a product centre from the
// pair's centre C) it follows from |CC'| >= E_ab(tau) + E_cd(tau),
// E(tau) = max_i r_i + tau (s_i / (2c) + c/4), tau = sqrt(tmin).  E is convex
// in tau: the pair stores it at FAR_TAU0 and FAR_TAU1, and the chord bounds
// it in between.  FAR_C2 is twice the 1/p of diffuse STO-nG pairs, where the
// tangent is tight.  Written in rounding intrinsics so that the two kernels
// that share a list decide alike; E covers the centres' rounding to float (of
// molecules far from the origin), the margin that of the test itself.
constexpr float FAR_C2 = 5.0f, FAR_TAU0 = 4.0f, FAR_TAU1 = 7.2f;

template <typename R, int L> __device__ __forceinline__ float far_extent(float e0, float e1) {
  constexpr float tm = far_tmin<R>(L);
  // sqrt(tmin) to 1e-4 from above (Newton from 6.1)
  constexpr float y = 0.5f * (6.1f + tm / 6.1f), z = 0.5f * (y + tm / y), tau = 1.0001f * z;
  static_assert(tau >= FAR_TAU0 && tau <= FAR_TAU1, "E is stored between these");
  constexpr float w = (tau - FAR_TAU0) / (FAR_TAU1 - FAR_TAU0);
  return __fmaf_rn(w, __fsub_rn(e1, e0), e0);
}

// a, b: {C, E(FAR_TAU0)}; ea, eb: far_extent of the pairs.
__device__ __forceinline__ bool far_pair(const float4& a, float ea, const float4& b, float eb) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
  const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
  const float need = __fadd_rn(__fadd_rn(ea, eb), 2e-3f);
  return d2 >= __fmul_rn(need, need);
}

// 1/sqrt(x) of a normal positive double: the hardware estimate y and the
// binomial series of (1 - e)^(-1/2), e = 1 - x y^2, to second order:
// y (1 + e/2 + 3 e^2/8), what is left out 5/16 e^3, below 2^-58 for the
// estimate's 2^-19.
__device__ __forceinline__ double far_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ F2 far_rsqrt(F2 x) {
  float a, b;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(x.v.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(x.v.y));
  return F2(a, b);
}
__device__ __forceinline__ float far_rsqrt(float x) {
  float a;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(x));
  return a;
}

// Quantities of a far primitive quartet in the form of PrimGeo; T is double,
// float or F2.  kk = k_ab k_cd, o2p = 1/(2p), o2q = 1/(2q).
template <typename T, int LM>
__device__ __forceinline__ void far_setup(const T PQ[3], T kk, T o2p, T o2q, PrimGeo<T>& g) {
  const T r2 = pf_fma(PQ[0], PQ[0], pf_fma(PQ[1], PQ[1], PQ[2] * PQ[2]));
  const T ri = far_rsqrt(r2);
  g.I[0] = kk * ri;
  if constexpr (LM > 0) {
    const T h = ri * ri * T(0.5f);
#pragma unroll
    for (int m = 1; m <= LM; ++m) g.I[m] = g.I[m - 1] * h * T((float)(2 * m - 1));
    g.nrp = o2p * T(-2.0f);
    g.nrq = o2q * T(-2.0f);
    const T ip = o2q * T(2.0f);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      g.WP[x] = g.nrp * PQ[x];
      g.WQ[x] = ip * PQ[x];
    }
    g.o2p = o2p;
    g.o2q = o2q;
    g.o2pq = o2p * ip;
  }
}

}  // namespace pyfacc

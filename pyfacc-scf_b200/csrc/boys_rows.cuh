// Boys function from a short table in shared memory, for the split kernels.
//
// boys_fp64 (boys.cuh) gathers four 16-byte pairs per lane from global memory,
// 2.6 wavefronts a quarter warp each (from rows of 64 bytes, as they were when
// this table was made, 5; the (ss|ss) kernel then spent 54 of its 63
// wavefronts per primitive quartet there).  Here F_L(T) on
// [0, 31.5 h) is one of 32 polynomials about T = k h, stored coefficient by
// coefficient, 32 words in 32 banks: a 4-byte load is conflict-free whatever
// rows the lanes want (one wavefront; an FP64 coefficient takes two, high and
// low word).  Longer intervals than boys.cuh's 0.1 cost 13 coefficients
// instead of 8.  Above the table F_L is its asymptote (far.cuh's bound), and
// the lower orders follow from the downward recursion with e^{-T}.
#pragma once
#include <cuda_runtime.h>

#include "far.cuh"

namespace pyfacc {

constexpr int BR_ROWS = 32;
constexpr int BR_N64 = 13;  // coefficients, FP64: interpolation error < 3e-17 F_L
constexpr int BR_N32 = 6;   // FP32: < 2e-8 F_L
constexpr int BR_LMAX = 4;

template <typename R> struct BoysRows;
template <> struct BoysRows<double> {
  unsigned hi[BR_N64][BR_ROWS], lo[BR_N64][BR_ROWS];
};
template <> struct BoysRows<float> {
  float c[BR_N32][BR_ROWS];
};
template <typename R> __host__ __device__ constexpr double br_step(int L) { return far_tmin<R>(L) / 31.5; }

// e^{-T}, 0 beyond T = 100: T = n ln 2 + r with the two-part ln 2 of Cody and
// Waite, e^{-r} by the degree-11 polynomial that interpolates it at the
// Chebyshev points of |r| <= ln(2)/2 (error < 2e-17).
__device__ __forceinline__ double br_expm(double T) {
  const double b = fma(T, 1.4426950408889634, 6755399441055744.0);
  const double n = b - 6755399441055744.0;
  const double r = fma(n, -7.440617110012397e-11, fma(n, -0.6931471804855391, T));
  double e = -2.5110037605963777e-08;
  e = fma(e, r, 2.763263963904103e-07);
  e = fma(e, r, -2.755724091857897e-06);
  e = fma(e, r, 2.4801485482328494e-05);
  e = fma(e, r, -0.00019841269890047113);
  e = fma(e, r, 0.0013888888952314775);
  e = fma(e, r, -0.008333333333319601);
  e = fma(e, r, 0.0416666666664881);
  e = fma(e, r, -0.1666666666666668);
  e = fma(e, r, 0.5000000000000019);
  e = fma(e, r, -1.0);
  e = fma(e, r, 1.0);
  const double s = __hiloint2double((1023 - (__double2loint(b) & 0xff)) << 20, 0);
  return T < 100.0 ? e * s : 0.0;
}

// Branch-free: skipping the table when no lane needs it (or the asymptote when
// all do) was 1-3% slower, as most warps hold both kinds.
template <int L>
__device__ __forceinline__ void boys_rows(const BoysRows<double>& tab, double T, double* __restrict__ F) {
  constexpr double h = br_step<double>(L);
  const double biased = fma(T, 1.0 / h, 6755399441055744.0);
  const int k = __double2loint(biased) & (BR_ROWS - 1);
  const double x = fma(biased - 6755399441055744.0, -h, T);
  double f = __hiloint2double(tab.hi[BR_N64 - 1][k], tab.lo[BR_N64 - 1][k]);
#pragma unroll
  for (int j = BR_N64 - 2; j >= 0; --j) f = fma(f, x, __hiloint2double(tab.hi[j][k], tab.lo[j][k]));
  const double rt = far_rsqrt(T);
  double fa = 0.88622692545275801365 * rt;
  const double o2t = 0.5 * rt * rt;
#pragma unroll
  for (int m = 0; m < L; ++m) fa = fa * o2t * (2 * m + 1);
  F[L] = T < 31.49 * h ? f : fa;  // (below the rounding to row 32)
  if constexpr (L > 0) {
    const double e = br_expm(T), t2 = 2.0 * T;
#pragma unroll
    for (int m = L - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], e) * (1.0 / (2 * m + 1));
  }
}

// Two arguments in a packed pair.
template <int L> __device__ __forceinline__ void boys_rows(const BoysRows<float>& tab, F2 T, F2* __restrict__ F) {
  constexpr float h = (float)br_step<float>(L), tmax = 31.49f * h;
  const F2 biased = pf_fma(T, F2(1.0f / h), F2(12582912.0f));
  const int kx = __float_as_int(biased.v.x) & (BR_ROWS - 1), ky = __float_as_int(biased.v.y) & (BR_ROWS - 1);
  const F2 x = pf_fma(biased + F2(-12582912.0f), F2(-h), T);
  F2 f(tab.c[BR_N32 - 1][kx], tab.c[BR_N32 - 1][ky]);
#pragma unroll
  for (int j = BR_N32 - 2; j >= 0; --j) f = pf_fma(f, x, F2(tab.c[j][kx], tab.c[j][ky]));
  const F2 rt = far_rsqrt(T);
  F2 fa = F2(0.88622692545275801365f) * rt;
  const F2 o2t = F2(0.5f) * rt * rt;
#pragma unroll
  for (int m = 0; m < L; ++m) fa = fa * o2t * F2((float)(2 * m + 1));
  F[L] = F2(T.v.x < tmax ? f.v.x : fa.v.x, T.v.y < tmax ? f.v.y : fa.v.y);
  if constexpr (L > 0) {
    const F2 e(expf(-T.v.x), expf(-T.v.y)), t2 = T + T;
#pragma unroll
    for (int m = L - 1; m >= 0; --m) F[m] = pf_fma(t2, F[m + 1], e) * F2(1.0f / (2 * m + 1));
  }
}

}  // namespace pyfacc

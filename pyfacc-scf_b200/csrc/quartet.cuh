// Device code shared by the kernels that evaluate s/p shell quartets
// (kernels.cu, jk_split.cu): the set-up of a primitive quartet, the
// contracted quartet of one lane, task search and density bounds.
#pragma once
#include <cuda_runtime.h>

#include "boys.cuh"
#include "engine.h"
#include "eri_classes.cuh"

namespace pyfacc {

// ---------------------------------------------------------------------------
// One primitive quartet: prefactors, Boys, VRR (shared by J/K, Schwarz,
// gradient and tensor kernels).
// ---------------------------------------------------------------------------
template <typename R>
struct PrimGeo {
  R I[PF_BOYS_MMAX + 1];
  R WP[3], WQ[3];
  R o2p, nrp, o2q, nrq, o2pq;  // nrp = -rho/p, nrq = -rho/q
};

template <typename R> struct Rec;  // primitive-pair record vector of a precision
template <> struct Rec<double> { using T = double4; };
template <> struct Rec<float> { using T = float4; };

// bra record b0..b2 and ket record k0..k2 (3 vectors each)
template <typename R, int LM, typename V>
__device__ __forceinline__ void prim_setup(const V& b0, const V& b1, const V& k0, const V& k1, PrimGeo<R>& g) {
  const R p = (R)b0.x, q = (R)k0.x;
  const R PQx = (R)(b1.x - k1.x), PQy = (R)(b1.y - k1.y), PQz = (R)(b1.z - k1.z);
  const R zeta = p + q;
  R rs, oz;
  if constexpr (sizeof(R) == 8) {
    rs = rsqrt((double)zeta);
  } else {
    rs = rsqrtf((float)zeta);
  }
  oz = rs * rs;
  const R rho = p * q * oz;
  const R T = rho * (PQx * PQx + PQy * PQy + PQz * PQz);
  const R pref = (R)b0.z * (R)k0.z * rs;
  R F[LM + 1];
  Boys<LM, R>::eval(T, F);
#pragma unroll
  for (int m = 0; m <= LM; ++m) g.I[m] = pref * F[m];
  const R qz = q * oz, pz = p * oz;
  g.WP[0] = -qz * PQx; g.WP[1] = -qz * PQy; g.WP[2] = -qz * PQz;
  g.WQ[0] = pz * PQx;  g.WQ[1] = pz * PQy;  g.WQ[2] = pz * PQz;
  g.o2p = (R)b0.y;
  g.o2q = (R)k0.y;
  g.nrp = -qz;  // -rho / p
  g.nrq = -pz;  // -rho / q
  g.o2pq = (R)0.5 * oz;
}

template <int L> struct NC { static constexpr int v = (L + 1) * (L + 2) / 2; };

// Contracted (ab|cd) for one bra pair and one ket pair (records of the
// kernel's precision: double4 for FP64 quartets, float4 for FP32 ones).
// Primitive pairs are stored in order of decreasing |K|, so with kcut > 0
// both loops stop at the first primitive quartet with |K_ab K_cd| < kcut.
// With kq_step > 1 only the ket primitives kq0, kq0 + kq_step, ... are
// summed, and of the bra's only kp0, kp0 + kp_step, ... (a share of the
// quartet; the shares add up to the integral).
// brec: the bra pair's first primitive record (in global memory, or the
// copy a warp staged in shared memory); prim: all records (the kets').
template <typename R, int LA, int LB, int LC, int LD>
__device__ __forceinline__ int contracted_quartet(const typename Rec<R>::T* __restrict__ prim,
                                                  const typename Rec<R>::T* brec, int4 bi0, int4 ki0,
                                                  const double4& bgeo, const double4& kgeo,
                                                  R out[EriClass<R, LA, LB, LC, LD>::NOUT], double kcut = 0.0,
                                                  int kq0 = 0, int kq_step = 1, int kp0 = 0, int kp_step = 1) {
  using C = EriClass<R, LA, LB, LC, LD>;
  using V = typename Rec<R>::T;
  R acc[C::NACC];
#pragma unroll
  for (int i = 0; i < C::NACC; ++i) acc[i] = (R)0;
  // the cut is compared in the records' precision (no FP64 work in the FP32
  // loop); a cut beyond the float range becomes +inf, which skips everything
  const R cut = (R)kcut;
  const R kab_max = fabs((R)brec[0].z);
  int nprim = 0;
  for (int kq = kq0; kq < ki0.w; kq += kq_step) {
    const V* kr = prim + 3 * (size_t)(ki0.z + kq);
    const V k0 = kr[0], k1 = kr[1], k2 = kr[2];
    const R kcd = fabs((R)k0.z);
    if (kab_max * kcd < cut) break;
    const R QC[3] = {(R)k2.x, (R)k2.y, (R)k2.z};
#pragma unroll 1
    for (int kp = kp0; kp < bi0.w; kp += kp_step) {
      const V* br = brec + 3 * kp;
      const V b0 = br[0], b1 = br[1], b2 = br[2];
      if (fabs((R)b0.z) * kcd < cut) break;
      const R PA[3] = {(R)b2.x, (R)b2.y, (R)b2.z};
      PrimGeo<R> g;
      prim_setup<R, C::L>(b0, b1, k0, k1, g);
      C::vrr(g.I, PA, g.WP, QC, g.WQ, g.o2p, g.nrp, g.o2q, g.nrq, g.o2pq, acc);
      ++nprim;
    }
  }
  const R AB[3] = {(R)bgeo.x, (R)bgeo.y, (R)bgeo.z};
  const R CD[3] = {(R)kgeo.x, (R)kgeo.y, (R)kgeo.z};
  C::hrr(acc, AB, CD, out);
  return nprim;
}

// The FP32 contracted quartet with two bra primitives per step in packed
// float pairs (FFMA2, f2.cuh): the same primitive quartets, cuts and sums as
// contracted_quartet<float>, but each Obara-Saika step of the generated
// recursion does the work of both primitives in one instruction.  An odd
// bra primitive count, or a second primitive below the cut, fills the upper
// half with the lower primitive at zero weight.
template <int L>
__device__ __forceinline__ void prim_setup_f2(const float4& blo0, const float4& blo1, const float4& bhi0,
                                              const float4& bhi1, float khi_weight, const float4& k0,
                                              const float4& k1, PrimGeo<F2>& g) {
  const F2 p(blo0.x, bhi0.x), q(k0.x);
  const F2 PQx = F2(blo1.x, bhi1.x) + F2(-k1.x), PQy = F2(blo1.y, bhi1.y) + F2(-k1.y),
           PQz = F2(blo1.z, bhi1.z) + F2(-k1.z);
  const F2 zeta = p + q;
  const F2 rs(rsqrtf(zeta.v.x), rsqrtf(zeta.v.y));
  const F2 oz = rs * rs;
  const F2 rho = p * q * oz;
  const F2 T = rho * pf_fma(PQx, PQx, pf_fma(PQy, PQy, PQz * PQz));
  const F2 pref = F2(blo0.z, bhi0.z * khi_weight) * F2(k0.z) * rs;
  F2 F[L + 1];
  boys_fp32x2<L>(T, F);
#pragma unroll
  for (int m = 0; m <= L; ++m) g.I[m] = pref * F[m];
  const F2 qz = q * oz, pz = p * oz;
  const F2 nqz = qz * F2(-1.0f);
  g.WP[0] = nqz * PQx; g.WP[1] = nqz * PQy; g.WP[2] = nqz * PQz;
  g.WQ[0] = pz * PQx;  g.WQ[1] = pz * PQy;  g.WQ[2] = pz * PQz;
  g.o2p = F2(blo0.y, bhi0.y);
  g.o2q = F2(k0.y);
  g.nrp = nqz;               // -rho / p
  g.nrq = pz * F2(-1.0f);    // -rho / q
  g.o2pq = F2(0.5f) * oz;
}

template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ int contracted_quartet_f2(const float4* __restrict__ prim, const float4* brec, int4 bi0,
                                                     int4 ki0, const double4& bgeo, const double4& kgeo,
                                                     float out[EriClass<float, LA, LB, LC, LD>::NOUT],
                                                     double kcut = 0.0, int kq0 = 0, int kq_step = 1, int kp0 = 0,
                                                     int kp_step = 1) {
  using C2 = EriClass<F2, LA, LB, LC, LD>;
  using C1 = EriClass<float, LA, LB, LC, LD>;
  F2 acc[C2::NACC];
#pragma unroll
  for (int i = 0; i < C2::NACC; ++i) acc[i] = F2(0.0f);
  const float cut = (float)kcut;
  const float kab_max = fabsf(brec[0].z);
  int nprim = 0;
  for (int kq = kq0; kq < ki0.w; kq += kq_step) {
    const float4* kr = prim + 3 * (size_t)(ki0.z + kq);
    const float4 k0 = kr[0], k1 = kr[1], k2 = kr[2];
    const float kcd = fabsf(k0.z);
    if (kab_max * kcd < cut) break;
    const F2 QC[3] = {F2(k2.x), F2(k2.y), F2(k2.z)};
#pragma unroll 1
    for (int kp = 2 * kp0; kp < bi0.w; kp += 2 * kp_step) {
      const float4* br = brec + 3 * kp;
      const float4 b0 = br[0], b1 = br[1], b2 = br[2];
      if (fabsf(b0.z) * kcd < cut) break;
      // the second primitive, or the first again at zero weight
      bool two = kp + 1 < bi0.w;
      float4 c0 = b0, c1 = b1, c2 = b2;
      if (two) {
        c0 = br[3];
        two = fabsf(c0.z) * kcd >= cut;
        if (two) {
          c1 = br[4];
          c2 = br[5];
        } else {
          c0 = b0;
        }
      }
      const F2 PA[3] = {F2(b2.x, c2.x), F2(b2.y, c2.y), F2(b2.z, c2.z)};
      PrimGeo<F2> g;
      prim_setup_f2<C2::L>(b0, b1, c0, c1, two ? 1.0f : 0.0f, k0, k1, g);
      C2::vrr(g.I, PA, g.WP, QC, g.WQ, g.o2p, g.nrp, g.o2q, g.nrq, g.o2pq, acc);
      nprim += two ? 2 : 1;
      if (!two) break;
    }
  }
  float accs[C1::NACC];
#pragma unroll
  for (int i = 0; i < C1::NACC; ++i) accs[i] = acc[i].v.x + acc[i].v.y;
  const float AB[3] = {(float)bgeo.x, (float)bgeo.y, (float)bgeo.z};
  const float CD[3] = {(float)kgeo.x, (float)kgeo.y, (float)kgeo.z};
  C1::hrr(accs, AB, CD, out);
  return nprim;
}

__device__ __forceinline__ int find_bra(const int* __restrict__ task_off, int nbra, int t) {
  int lo = 0, hi = nbra;  // task_off[lo] <= t < task_off[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (__ldg(task_off + mid) <= t) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float dmax_bound(const float* __restrict__ dm, int ld, int a, int b, int c, int d) {
  float m = 2.0f * fmaxf(__ldg(dm + a * ld + b), __ldg(dm + c * ld + d));
  m = fmaxf(m, __ldg(dm + a * ld + c));
  m = fmaxf(m, __ldg(dm + a * ld + d));
  m = fmaxf(m, __ldg(dm + b * ld + c));
  m = fmaxf(m, __ldg(dm + b * ld + d));
  return m;
}

}  // namespace pyfacc

// Two-electron nuclear gradient of long quartet lists, far and near quartets
// apart: the walk, the queues and the far limit of jk_split.cu, the derivatives
// (grad_md.cuh), the screening and the density products of grad2e_kernel
// (kernels.cu).  FP64 gradients of C40H82 10.2 -> 8.7 ms, C100H202 60 -> 53 ms,
// and with the Hermite derivatives 5.9 and 29.5; FP32 lists (two bra primitives
// at a time in packed pairs) only with the latter: mixed gradient of gly30 18.9
// -> 15.6 ms, C100H202 29.0 -> 18.2.
#include <cuda_runtime.h>

#include <algorithm>

#include "grad_md.cuh"
#include "split.cuh"

namespace pyfacc {

namespace {

struct GradSplitArgs {
  SplitLists l;
  GradArgs a;
  int smem_atoms;  // atoms summed in shared memory (0: global atomics)
};

// Staged bra records, twelve words a unit: {P, k}, {P-A, 1/2p}, {2 alpha,
// 2 beta, p, K}, then |K| in float.  A unit is one primitive pair in FP64 and
// two interleaved ones in FP32 (F2; an odd count is filled up with zero weight).
template <typename R> struct GradStage {
  static constexpr int WORDS = 12, UNIT = sizeof(R) == 8 ? 1 : 2;
  static __host__ __device__ constexpr int units(int n) { return (n + UNIT - 1) / UNIT; }
  static __host__ __device__ constexpr size_t bytes(int maxp) {
    return (size_t)units(maxp) * WORDS * 8 + (size_t)(maxp + 3) / 4 * 16;
  }
  __device__ static __forceinline__ float* kab(unsigned char* st, int maxp) {
    return reinterpret_cast<float*>(st + (size_t)units(maxp) * WORDS * 8);
  }
};

__device__ __forceinline__ int stage_grad_bra(const SplitLists& l, const int4& bi0, double, unsigned char* st, int lane) {
  const double4* br = l.prim + 3 * (size_t)bi0.z;
  double4* v = reinterpret_cast<double4*>(st);
  float* kab = GradStage<double>::kab(st, l.maxp);
  for (int i = lane; i < bi0.w; i += 32) {
    const double4 r0 = br[3 * i];
    kab[i] = fabsf((float)r0.z);
    v[3 * i] = br[3 * i + 1];
    v[3 * i + 1] = br[3 * i + 2];
    v[3 * i + 2] = make_double4(2 * r0.w, 2 * (r0.x - r0.w), r0.x, r0.z);
  }
  return bi0.w;
}
__device__ __forceinline__ int stage_grad_bra(const SplitLists& l, const int4& bi0, float, unsigned char* st, int lane) {
  const float4* br = l.primf + 3 * (size_t)bi0.z;
  float* kab = GradStage<float>::kab(st, l.maxp);
  for (int i = lane; i < 2 * GradStage<float>::units(bi0.w); i += 32) {
    const int s = min(i, bi0.w - 1);
    const float w = i < bi0.w ? 1.0f : 0.0f;
    const float4 r0 = br[3 * s], r1 = br[3 * s + 1], r2 = br[3 * s + 2];
    if (i < bi0.w) kab[i] = fabsf(r0.z);
    float* o = reinterpret_cast<float*>(st) + (size_t)(i >> 1) * 24 + (i & 1);
    o[0] = r1.x; o[2] = r1.y; o[4] = r1.z; o[6] = w * r1.w;
    o[8] = r2.x; o[10] = r2.y; o[12] = r2.z; o[14] = r2.w;
    o[16] = 2.0f * r0.w; o[18] = 2.0f * (r0.x - r0.w); o[20] = r0.x; o[22] = w * r0.z;
  }
  return bi0.w;
}

template <bool FAR>
__device__ __forceinline__ void load_grad_unit(const unsigned char* st, int i, PrimSide<double>& b, double& ta, double& tb) {
  const double4* v = reinterpret_cast<const double4*>(st) + 3 * i;
  const double4 b0 = v[0], b1 = v[1], b2 = v[2];
  b.P[0] = b0.x; b.P[1] = b0.y; b.P[2] = b0.z;
  b.A[0] = b1.x; b.A[1] = b1.y; b.A[2] = b1.z;
  b.o2p = b1.w;
  ta = b2.x;
  tb = b2.y;
  b.p = b2.z;
  b.k = FAR ? b0.w : b2.w;
}
template <bool FAR>
__device__ __forceinline__ void load_grad_unit(const unsigned char* st, int i, PrimSide<F2>& b, F2& ta, F2& tb) {
  const float4* v = reinterpret_cast<const float4*>(st) + 6 * i;
  const float4 a0 = v[0], a1 = v[1], c0 = v[2], c1 = v[3], e0 = v[4], e1 = v[5];
  b.P[0] = F2(a0.x, a0.y); b.P[1] = F2(a0.z, a0.w); b.P[2] = F2(a1.x, a1.y);
  b.A[0] = F2(c0.x, c0.y); b.A[1] = F2(c0.z, c0.w); b.A[2] = F2(c1.x, c1.y);
  b.o2p = F2(c1.z, c1.w);
  ta = F2(e0.x, e0.y);
  tb = F2(e0.z, e0.w);
  b.p = F2(e1.x, e1.y);
  b.k = FAR ? F2(a1.z, a1.w) : F2(e1.z, e1.w);
}
// The ket's exponents, doubled (an F2 ket has the same primitive twice).
__device__ __forceinline__ void ket_exponents(double al, double o2p, double& tc, double& td) {
  tc = 2.0 * al;
  td = 1.0 / o2p - tc;
}
__device__ __forceinline__ void ket_exponents(double al, F2 o2p, F2& tc, F2& td) {
  const float c = (float)(2.0 * al);
  tc = F2(c);
  td = F2(1.0f / o2p.v.x - c);
}
__device__ __forceinline__ double whole(double a) { return a; }
__device__ __forceinline__ double whole(F2 a) { return (double)(a.v.x + a.v.y); }

// Resident blocks per SM that the registers are held to (5 / 3 / 2 / 2 for
// L = 0 / 1 / 2 / 3: gly30 26.6 instead of 25.3 ms).
__host__ __device__ constexpr int grad_min_blocks(int L) { return L < 2 ? 4 : (L == 2 ? 3 : 2); }

template <typename R, int LA, int LB, int LC, int LD, bool FAR>
__global__ void __launch_bounds__(128, grad_min_blocks(LA + LB + LC + LD)) grad_split_kernel(const GradSplitArgs args) {
  using C = EriClass<R, LA, LB, LC, LD>;
  using S = GradStage<R>;
  using T = typename std::conditional<sizeof(R) == 8, double, F2>::type;
  constexpr int NA = NC<LA>::v, NB = NC<LB>::v, NCc = NC<LC>::v, ND = NC<LD>::v, LM = C::L + 1;
  extern __shared__ __align__(16) unsigned char gsplit_smem[];
  __shared__ int2 queue[4][1][QUEUE];
  __shared__ int2 slot_bra[4][MAXSLOT];
  __shared__ typename std::conditional<FAR, int, BoysRows<R>>::type tab_smem;
  const BoysRows<R>& tab = reinterpret_cast<const BoysRows<R>&>(tab_smem);  // near half only
  const SplitLists& L = args.l;
  const GradArgs& A = args.a;
  double* gsh = reinterpret_cast<double*>(gsplit_smem);
  const int nsm = 3 * args.smem_atoms;
  if constexpr (!FAR) {
    const unsigned* src = static_cast<const unsigned*>(L.boys);
    unsigned* dst = reinterpret_cast<unsigned*>(&tab_smem);
    for (int i = threadIdx.x; i < (int)(sizeof(BoysRows<R>) / 4); i += blockDim.x) dst[i] = src[i];
  }
  for (int i = threadIdx.x; i < nsm; i += blockDim.x) gsh[i] = 0.0;
  __syncthreads();
  double* G = nsm ? gsh : A.grad;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const size_t slot_bytes = S::bytes(L.maxp);
  unsigned char* st = gsplit_smem + ((size_t)nsm * sizeof(double) + 15) / 16 * 16 + (size_t)wib * L.nslot * slot_bytes;
  int nquart = 0;
  unsigned nprim = 0;
  // the bra's part of the gradient stays in registers while the bra does
  double sum[6] = {0, 0, 0, 0, 0, 0};
  int sum_a = -1, sum_b = -1;
  auto flush = [&]() {
    if (sum_a < 0) return;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const double sa = warp_sum(sum[x]), sb = warp_sum(sum[3 + x]);
      if (lane == 0) {
        atomicAdd(G + 3 * sum_a + x, sa);
        atomicAdd(G + 3 * sum_b + x, sb);
      }
      sum[x] = sum[3 + x] = 0.0;
    }
  };
  auto stage = [&](int ib, int slot) {
    return stage_grad_bra(L, L.info0[L.bra_base + ib], (R)0, st + slot * slot_bytes, lane);
  };
  auto test = [&](int ib, int ket, float& cut) {
    const int bp = L.bra_base + ib, kp = L.ket_base + ket;
    const float4 bc = L.test[bp], bt = L.test2[bp], kc = L.test[kp], kt = L.test2[kp];
    if ((FAR || L.halves) &&
        far_pair(bc, far_extent<R, LM>(bc.w, bt.x), kc, far_extent<R, LM>(kc.w, kt.x)) != FAR)
      return -1;
    if (A.dmax) {
      const float* dmx = A.dmax + L.info2[bp].w;
      const float dm = dmax_bound(dmx, A.ns_ld, __float_as_int(bt.z), __float_as_int(bt.w), __float_as_int(kt.z),
                                  __float_as_int(kt.w));
      if (!(bt.y * kt.y * dm >= TEST_SLACK * (float)A.thresh)) return -1;
      if (A.prim_thresh > 0.0) cut = TEST_SLACK * __fdividef((float)A.prim_thresh, fmaxf(dm, 1e-30f));
    }
    return 0;
  };
  auto eval = [&](int, const Queued& q) {
    const int bp = L.bra_base + q.bra.x, kp = L.ket_base + q.ket;
    const int4 bi1 = L.info1[bp], ki1 = L.info1[kp];
    double g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (q.active) {
      const int4 bi0 = L.info0[bp], ki0 = L.info0[kp], bi2 = L.info2[bp];
      const int ld = bi2.y, ma = bi0.x, mb = bi0.y, mc = ki0.x, md = ki0.y;
      const double4 bg = L.geom[bp], kg = L.geom[kp];
      const T AB[3] = {T((R)bg.x), T((R)bg.y), T((R)bg.z)}, CD[3] = {T((R)kg.x), T((R)kg.y), T((R)kg.z)};
      auto fill_gam = [&](R* gam) {
        const double* Pt = A.Pt + bi2.x;
        const double* Pa = A.Pa + bi2.x;
        const double* Pb = A.Pb + bi2.x;
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int c = 0; c < NCc; ++c)
#pragma unroll
              for (int d = 0; d < ND; ++d) {
                const int mu = (ma + a) * ld, nu = (mb + b) * ld, la = mc + c, si = md + d;
                double v = __ldg(Pt + mu + mb + b) * __ldg(Pt + la * ld + si);
                if (A.uhf) {
                  v -= 0.5 * (__ldg(Pa + mu + la) * __ldg(Pa + nu + si) + __ldg(Pa + mu + si) * __ldg(Pa + nu + la));
                  v -= 0.5 * (__ldg(Pb + mu + la) * __ldg(Pb + nu + si) + __ldg(Pb + mu + si) * __ldg(Pb + nu + la));
                } else {
                  v -= 0.25 * (__ldg(Pt + mu + la) * __ldg(Pt + nu + si) + __ldg(Pt + mu + si) * __ldg(Pt + nu + la));
                }
                gam[((a * NB + b) * NCc + c) * ND + d] = (R)v;
              }
      };
      unsigned char* sb = st + q.slot * slot_bytes;
      const float* kab = S::kab(sb, L.maxp);
      T gr[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) gr[i] = T(0.0f);
      R gam[C::NOUT];
      fill_gam(gam);
      int n = q.bra.y, np = 0;
#pragma unroll 1
      for (int kq = 0; kq < ki0.w; ++kq) {
        const size_t sl = (size_t)kq * L.nket + q.ket;
        const float kcd = L.ket.kabs[sl];
        PrimSide<T> k;
        load_ket<true, FAR>(L.ket, sl, k);
        T tc, td;
        ket_exponents(L.ket.al[sl], k.o2p, tc, td);
        MdSide<T> ks;
        md_side(k.A, CD, k.o2p, tc, td, ks);
        while (n > 0 && kab[n - 1] * kcd < q.cut) --n;
        if (n == 0) break;
        np += n;
        const int nu = S::units(n);
#pragma unroll 1
        for (int i = 0; i < nu; ++i) {
          PrimSide<T> b;
          T ta, tb, PQ[3];
          load_grad_unit<FAR>(sb, i, b, ta, tb);
#pragma unroll
          for (int x = 0; x < 3; ++x) PQ[x] = b.P[x] + k.P[x] * T(-1.0f);
          PrimGeo<T> pg;
          if constexpr (FAR) far_setup<T, LM>(PQ, b.k * k.k, b.o2p, k.o2p, pg);
          else near_setup<T, LM>(tab, PQ, b, k, pg);
          MdSide<T> bs;
          md_side(b.A, AB, b.o2p, ta, tb, bs);
          md_gradient<T, LA + LB, LC + LD>(
              pg.I, FAR ? T(-2.0f) : T(2.0f) * pg.nrp * b.p, PQ, bs, ks,
              [&](int i, int j, int c, int d) { return T(gam[((i * NB + j) * NCc + c) * ND + d]); }, gr);
        }
      }
      nprim += np;
      ++nquart;
      double fac = 4.0;
      if (bi1.x == bi1.y) fac *= 0.5;
      if (ki1.x == ki1.y) fac *= 0.5;
      if (L.same_class && bp == kp) fac *= 0.5;
#pragma unroll
      for (int i = 0; i < 9; ++i) g[i] = fac * whole(gr[i]);
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        atomicAdd(G + 3 * ki1.z + x, g[6 + x]);
        atomicAdd(G + 3 * ki1.w + x, -(g[x] + g[3 + x] + g[6 + x]));
      }
    }
    const int a0 = __shfl_sync(0xffffffffu, bi1.z, 0), b0 = __shfl_sync(0xffffffffu, bi1.w, 0);
    if (q.one_bra) {
      if (a0 != sum_a || b0 != sum_b) {
        flush();
        sum_a = a0;
        sum_b = b0;
      }
#pragma unroll
      for (int x = 0; x < 6; ++x) sum[x] += g[x];
    } else if (q.active) {
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        atomicAdd(G + 3 * bi1.z + x, g[x]);
        atomicAdd(G + 3 * bi1.w + x, g[3 + x]);
      }
    }
  };
  split_run<1>(L, queue[wib], slot_bra[wib], stage, test, eval);
  flush();
  if (A.stats) {  // contracted and evaluated primitive quartets
    unsigned long long nq = (unsigned)nquart, p = nprim;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nq += __shfl_xor_sync(0xffffffffu, nq, o);
      p += __shfl_xor_sync(0xffffffffu, p, o);
    }
    if (lane == 0 && nq) {
      unsigned long long* out = A.stats + (FAR ? GRAD_STATS_FAR : 0) + L.qclass;
      atomicAdd(out, nq);
      atomicAdd(out + NQCLASS, p);
    }
  }
  if (nsm) {
    __syncthreads();
    for (int i = threadIdx.x; i < nsm; i += blockDim.x)
      if (gsh[i] != 0.0) atomicAdd(A.grad + i, gsh[i]);
  }
}

constexpr size_t GRAD_STAGE_MAX_BYTES = 24 * 1024;
constexpr int GRAD_SPLIT_SMEM_ATOMS = 1024;  // 24 KB a block

template <typename R, int LA, int LB, int LC, int LD, bool FAR>
void launch_one(int num_sms, cudaStream_t s, GradSplitArgs k) {
  const size_t b = GradStage<R>::bytes(k.l.maxp);
  k.l.nslot = MAXSLOT;
  while (k.l.nslot > 2 && 4 * k.l.nslot * b > GRAD_STAGE_MAX_BYTES) k.l.nslot /= 2;
  const size_t smem = (3 * (size_t)k.smem_atoms * sizeof(double) + 15) / 16 * 16 + 4 * k.l.nslot * b;
  if (smem > 32 * 1024)
    allow_smem(grad_split_kernel<R, LA, LB, LC, LD, FAR>,
               3 * GRAD_SPLIT_SMEM_ATOMS * sizeof(double) +
                   std::max(GRAD_STAGE_MAX_BYTES, 4 * 2 * GradStage<R>::bytes(SPLIT_MAXPRIM)));
  const int blocks = (int)std::max(
      1LL, std::min((k.l.ntasks + 3LL) / 4, (long long)num_sms * grad_min_blocks(LA + LB + LC + LD)));
  grad_split_kernel<R, LA, LB, LC, LD, FAR><<<blocks, 128, smem, s>>>(k);
  PF_CUDA(cudaGetLastError());
  count_split_launch(FAR);
}

template <typename R, int LA, int LB, int LC, int LD>
void launch_halves(int num_sms, cudaStream_t s_far, cudaStream_t s_near, GradSplitArgs k) {
  launch_one<R, LA, LB, LC, LD, false>(num_sms, s_near, k);
  ++k.l.next;
  if (k.l.halves) launch_one<R, LA, LB, LC, LD, true>(num_sms, s_far, k);
}

template <typename R>
void dispatch(int num_sms, cudaStream_t s_far, cudaStream_t s_near, const GradSplitArgs& k) {
  switch (k.l.qclass) {
    case 0: launch_halves<R, 0, 0, 0, 0>(num_sms, s_far, s_near, k); break;
    case 1: launch_halves<R, 1, 0, 0, 0>(num_sms, s_far, s_near, k); break;
    case 2: launch_halves<R, 1, 0, 1, 0>(num_sms, s_far, s_near, k); break;
    case 3: launch_halves<R, 1, 1, 0, 0>(num_sms, s_far, s_near, k); break;
    default: launch_halves<R, 1, 1, 1, 0>(num_sms, s_far, s_near, k); break;
  }
}

}  // namespace

void launch_grad_split(const PairData& pd, const TaskList& tl, int bc, int kc, bool fp32, const GradArgs& a,
                       int num_sms, int* next, cudaStream_t s_far, cudaStream_t s_near) {
  if (tl.ntasks_c <= 0) return;
  if (fp32 && !pd.primf) throw Error(PYFACC_ERR_INVALID, "FP32 quartets need float primitive records");
  GradSplitArgs k{};
  k.l = split_lists(pd, tl, bc, kc, next);
  k.l.boys = boys_rows_table(fp32, class_flops(k.l.qclass).L + 1);
  k.a = a;
  // the resident blocks flush once: atoms that the kets scatter to are summed in
  // shared memory as far as it reaches (C100H202, 302 atoms: FP64 gradient 37.6 ->
  // 28.6 ms, mixed 28.4 -> 17.5; launch_grad2e's line is 256)
  k.smem_atoms = (a.natoms_total > 0 && a.natoms_total <= GRAD_SPLIT_SMEM_ATOMS) ? a.natoms_total : 0;
  if (fp32) dispatch<float>(num_sms, s_far, s_near, k);
  else dispatch<double>(num_sms, s_far, s_near, k);
}

}  // namespace pyfacc

// Two-electron nuclear gradient of long quartet lists, far and near quartets
// apart: the walk, the queues and the far limit of jk_split.cu, the derivatives
// (grad_md.cuh) and the density products of grad2e_kernel (kernels.cu).  A quartet is left out when Q_ab Q_cd times the bound on its
// density products, |D_ab D_cd| + |D_ac D_bd| + |D_ad D_bc|, stays below
// GRAD_SPLIT_REL of the screening threshold: the undivided kernels test one
// density factor, the largest, and evaluate quartets whose products are orders
// of magnitude smaller.  FP64 only: C40H82 10.2 -> 8.6 ms, C100H202 60 -> 52 ms
// (with the generated derivative routines of the time), max |dg| against the
// undivided kernels 1e-11 Ha/bohr; in FP32 the split gained 0-5%.
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

// Staged bra records, one primitive pair each: {P, k}, {P-A, 1/2p}, {2 alpha,
// 2 beta, p, K}, then |K| in float.
struct GradStage {
  static constexpr int WORDS = 12;
  static __host__ __device__ constexpr size_t bytes(int maxp) {
    return (size_t)maxp * WORDS * sizeof(double) + (size_t)(maxp + 3) / 4 * 16;
  }
  __device__ static __forceinline__ float* kab(unsigned char* st, int maxp) {
    return reinterpret_cast<float*>(st + (size_t)maxp * WORDS * sizeof(double));
  }
};

__device__ __forceinline__ int stage_grad_bra(const SplitLists& l, const int4& bi0, unsigned char* st, int lane) {
  const double4* br = l.prim + 3 * (size_t)bi0.z;
  double4* v = reinterpret_cast<double4*>(st);
  float* kab = GradStage::kab(st, l.maxp);
  for (int i = lane; i < bi0.w; i += 32) {
    const double4 r0 = br[3 * i];
    kab[i] = fabsf((float)r0.z);
    v[3 * i] = br[3 * i + 1];
    v[3 * i + 1] = br[3 * i + 2];
    v[3 * i + 2] = make_double4(2 * r0.w, 2 * (r0.x - r0.w), r0.x, r0.z);
  }
  return bi0.w;
}

template <bool FAR>
__device__ __forceinline__ void load_grad_ket(const KetTables& t, size_t sl, PrimSide<double>& k, double& tc) {
  load_ket<true, FAR>(t, sl, k);
  tc = 2 * t.al[sl];
}
// Resident blocks per SM that the registers are held to (5 / 3 / 2 / 2 for
// L = 0 / 1 / 2 / 3: gly30 26.6 instead of 25.3 ms).
__host__ __device__ constexpr int grad_min_blocks(int L) { return L < 2 ? 4 : (L == 2 ? 3 : 2); }

template <int LA, int LB, int LC, int LD, bool FAR>
__global__ void __launch_bounds__(128, grad_min_blocks(LA + LB + LC + LD)) grad_split_kernel(const GradSplitArgs args) {
  using C = EriClass<double, LA, LB, LC, LD>;
  constexpr int NA = NC<LA>::v, NB = NC<LB>::v, NCc = NC<LC>::v, ND = NC<LD>::v, LM = C::L + 1;
  extern __shared__ __align__(16) unsigned char gsplit_smem[];
  __shared__ int2 queue[4][1][QUEUE];
  __shared__ int2 slot_bra[4][MAXSLOT];
  __shared__ typename std::conditional<FAR, int, BoysRows<double>>::type tab_smem;
  const BoysRows<double>& tab = reinterpret_cast<const BoysRows<double>&>(tab_smem);  // near half only
  const SplitLists& L = args.l;
  const GradArgs& A = args.a;
  double* gsh = reinterpret_cast<double*>(gsplit_smem);
  const int nsm = 3 * args.smem_atoms;
  if constexpr (!FAR) {
    const unsigned* src = static_cast<const unsigned*>(L.boys);
    unsigned* dst = reinterpret_cast<unsigned*>(&tab_smem);
    for (int i = threadIdx.x; i < (int)(sizeof(BoysRows<double>) / 4); i += blockDim.x) dst[i] = src[i];
  }
  for (int i = threadIdx.x; i < nsm; i += blockDim.x) gsh[i] = 0.0;
  __syncthreads();
  double* G = nsm ? gsh : A.grad;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const size_t slot_bytes = GradStage::bytes(L.maxp);
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
    return stage_grad_bra(L, L.info0[L.bra_base + ib], st + slot * slot_bytes, lane);
  };
  auto test = [&](int ib, int ket, float& cut) {
    const int bp = L.bra_base + ib, kp = L.ket_base + ket;
    const float4 bc = L.test[bp], bt = L.test2[bp], kc = L.test[kp], kt = L.test2[kp];
    if ((FAR || L.halves) &&
        far_pair(bc, far_extent<double, LM>(bc.w, bt.x), kc, far_extent<double, LM>(kc.w, kt.x)) != FAR)
      return -1;
    if (A.dmax) {
      const float* dmx = A.dmax + L.info2[bp].w;
      const int ld = A.ns_ld, sa = __float_as_int(bt.z), sb = __float_as_int(bt.w), sc = __float_as_int(kt.z),
                sd = __float_as_int(kt.w);
      const float dab = __ldg(dmx + sa * ld + sb), dcd = __ldg(dmx + sc * ld + sd), dac = __ldg(dmx + sa * ld + sc),
                  dad = __ldg(dmx + sa * ld + sd), dbc = __ldg(dmx + sb * ld + sc), dbd = __ldg(dmx + sb * ld + sd);
      const float dm = fmaxf(fmaxf(2.0f * fmaxf(dab, dcd), fmaxf(dac, dad)), fmaxf(dbc, dbd));
      const float gm = dab * dcd + dac * dbd + dad * dbc, qq = bt.y * kt.y;
      if (!(qq * dm >= (float)A.thresh) || !(qq * gm >= (float)(GRAD_SPLIT_REL * A.thresh))) return -1;
      if (A.prim_thresh > 0.0) cut = __fdividef((float)A.prim_thresh, fmaxf(dm, 1e-30f));
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
      const double AB[3] = {bg.x, bg.y, bg.z}, CD[3] = {kg.x, kg.y, kg.z};
      auto fill_gam = [&](double* gam) {
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
                gam[((a * NB + b) * NCc + c) * ND + d] = v;
              }
      };
      const unsigned char* sb = st + q.slot * slot_bytes;
      const double4* bra = reinterpret_cast<const double4*>(sb);
      const float* kab = GradStage::kab(st + q.slot * slot_bytes, L.maxp);
      double gr[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      double acc[C::L == 0 ? C::NGACC : C::NOUT];  // accumulators, or the density products
      if constexpr (C::L == 0) {
#pragma unroll
        for (int i = 0; i < C::NGACC; ++i) acc[i] = 0.0;
      } else {
        fill_gam(acc);
      }
      int n = q.bra.y, np = 0;
#pragma unroll 1
      for (int kq = 0; kq < ki0.w; ++kq) {
        const size_t sl = (size_t)kq * L.nket + q.ket;
        const float kcd = L.ket.kabs[sl];
        PrimSide<double> k;
        double tc;
        load_grad_ket<FAR>(L.ket, sl, k, tc);
        while (n > 0 && kab[n - 1] * kcd < q.cut) --n;
        if (n == 0) break;
        np += n;
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
          const auto b0 = bra[3 * i], b1 = bra[3 * i + 1], b2 = bra[3 * i + 2];
          PrimSide<double> b;
          b.P[0] = b0.x; b.P[1] = b0.y; b.P[2] = b0.z;
          b.A[0] = b1.x; b.A[1] = b1.y; b.A[2] = b1.z;
          b.o2p = b1.w;
          double PQ[3];
#pragma unroll
          for (int x = 0; x < 3; ++x) PQ[x] = b.P[x] - k.P[x];
          PrimGeo<double> pg;
          if constexpr (FAR) {
            far_setup<double, LM>(PQ, b0.w * k.k, b.o2p, k.o2p, pg);
          } else {
            b.p = b2.z;
            b.k = b2.w;
            near_setup<double, LM>(tab, PQ, b, k, pg);
          }
          if constexpr (C::L == 0) {
            C::gacc(pg.I, b.A, pg.WP, k.A, pg.WQ, pg.o2p, pg.nrp, pg.o2q, pg.nrq, pg.o2pq, b2.x, b2.y, tc, acc);
          } else {
            MdSide<double> bs, ks;
            md_side(b.A, AB, b.o2p, b2.x, b2.y, bs);
            md_side(k.A, CD, k.o2p, tc, 1.0 / k.o2p - tc, ks);
            md_gradient<double, NB == 3, LC + LD>(
                pg.I, FAR ? -2.0 : 2.0 * pg.nrp * b2.z, PQ, bs, ks,
                [&](int i, int j, int c, int d) { return acc[((i * NB + j) * NCc + c) * ND + d]; }, gr);
          }
        }
      }
      if constexpr (C::L == 0) {
        double gam[C::NOUT];
        fill_gam(gam);
        C::gfin(acc, AB, CD, gam, gr);
      }
      nprim += np;
      ++nquart;
      double fac = 4.0;
      if (bi1.x == bi1.y) fac *= 0.5;
      if (ki1.x == ki1.y) fac *= 0.5;
      if (L.same_class && bp == kp) fac *= 0.5;
#pragma unroll
      for (int i = 0; i < 9; ++i) g[i] = fac * gr[i];
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
      atomicAdd(A.stats + L.qclass, nq);
      atomicAdd(A.stats + NQCLASS + L.qclass, p);
    }
  }
  if (nsm) {
    __syncthreads();
    for (int i = threadIdx.x; i < nsm; i += blockDim.x)
      if (gsh[i] != 0.0) atomicAdd(A.grad + i, gsh[i]);
  }
}

constexpr size_t GRAD_STAGE_MAX_BYTES = 24 * 1024;

template <int LA, int LB, int LC, int LD, bool FAR>
void launch_one(int num_sms, cudaStream_t s, GradSplitArgs k) {
  const size_t b = GradStage::bytes(k.l.maxp);
  k.l.nslot = MAXSLOT;
  while (k.l.nslot > 2 && 4 * k.l.nslot * b > GRAD_STAGE_MAX_BYTES) k.l.nslot /= 2;
  const size_t smem = (3 * (size_t)k.smem_atoms * sizeof(double) + 15) / 16 * 16 + 4 * k.l.nslot * b;
  if (smem > 32 * 1024)
    PF_CUDA(cudaFuncSetAttribute(grad_split_kernel<LA, LB, LC, LD, FAR>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int blocks = (int)std::max(
      1LL, std::min((k.l.ntasks + 3LL) / 4, (long long)num_sms * grad_min_blocks(LA + LB + LC + LD)));
  grad_split_kernel<LA, LB, LC, LD, FAR><<<blocks, 128, smem, s>>>(k);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

template <int LA, int LB, int LC, int LD>
void launch_halves(int num_sms, cudaStream_t s_far, cudaStream_t s_near, GradSplitArgs k) {
  launch_one<LA, LB, LC, LD, false>(num_sms, s_near, k);
  ++k.l.next;
  if (k.l.halves) launch_one<LA, LB, LC, LD, true>(num_sms, s_far, k);
}

void dispatch(int num_sms, cudaStream_t s_far, cudaStream_t s_near, const GradSplitArgs& k) {
  switch (k.l.qclass) {
    case 0: launch_halves<0, 0, 0, 0>(num_sms, s_far, s_near, k); break;
    case 1: launch_halves<1, 0, 0, 0>(num_sms, s_far, s_near, k); break;
    case 2: launch_halves<1, 0, 1, 0>(num_sms, s_far, s_near, k); break;
    case 3: launch_halves<1, 1, 0, 0>(num_sms, s_far, s_near, k); break;
    default: launch_halves<1, 1, 1, 0>(num_sms, s_far, s_near, k); break;
  }
}

}  // namespace

void launch_grad_split(const PairData& pd, const TaskList& tl, int bc, int kc, const GradArgs& a,
                       int num_sms, int* next, cudaStream_t s_far, cudaStream_t s_near) {
  if (tl.ntasks_c <= 0) return;
  GradSplitArgs k{};
  k.l = split_lists(pd, tl, bc, kc, next);
  k.l.boys = boys_rows_table(false, class_flops(k.l.qclass).L + 1);
  k.a = a;
  // as launch_grad2e: above 256 atoms the flush costs more than it saves
  k.smem_atoms = (a.natoms_total > 0 && a.natoms_total <= 256) ? a.natoms_total : 0;
  dispatch(num_sms, s_far, s_near, k);
}

}  // namespace pyfacc

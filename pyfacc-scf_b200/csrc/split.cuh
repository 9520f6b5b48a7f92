// Device code shared by the split kernels (jk_split.cu, grad_split.cu).
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "boys_rows.cuh"
#include "engine.h"
#include "far.cuh"
#include "quartet.cuh"

namespace pyfacc {

// What the split kernels' launches share: the lists, the pairs, their tests.
struct SplitLists {
  const int* ntasks_dev;
  const int4* info0;
  const int4* info1;
  const int4* info2;
  const double4* geom;
  const double4* prim;
  const float4* primf;
  const float4* test;   // {centre, extent} of all pairs
  const float4* test2;  // {extent, Q, shells}
  KetTables ket, bra;   // the classes' parts of the transposed records
  int nket, nbra_class, ketmaxp;
  const int* task_off;
  const int* ket_lo;
  const int* ket_hi;
  int nbra, ntasks, bra_base, bra_off, ket_base, same_class, qclass, task_begin;
  int chunk;  // kets per task (a multiple of 32)
  int halves; // 0: no far kernel, the near one takes every quartet
  int maxp;   // bra primitive pairs staged per run
  int nslot;  // runs staged at a time (a power of two)
  const void* boys;  // the class's BoysRows table
  int* next;  // tasks handed out beyond the first of every warp (zeroed)
};

// The lists' part of a launch, for a list that jk_splits.
inline SplitLists split_lists(const PairData& pd, const TaskList& tl, int bc, int kc, int* next) {
  SplitLists k{};
  k.ntasks_dev = tl.ntasks_dev;
  k.info0 = pd.info0; k.info1 = pd.info1; k.info2 = pd.info2;
  k.geom = pd.geom; k.prim = pd.prim; k.primf = pd.primf;
  k.test = pd.test; k.test2 = pd.test + pd.npair;
  k.ket = pd.kt.part(kc);
  k.bra = pd.kt.part(bc);
  k.nket = pd.class_off[kc + 1] - pd.class_off[kc];
  k.nbra_class = pd.class_off[bc + 1] - pd.class_off[bc];
  k.ketmaxp = pd.class_maxprim[kc];
  k.task_off = tl.off_c; k.ket_lo = tl.ket_lo; k.ket_hi = tl.ket_hi;
  k.nbra = tl.nbra; k.ntasks = tl.ntasks_c; k.task_begin = tl.task_begin_c;
  k.bra_base = pd.class_off[bc] + tl.bra_offset; k.bra_off = tl.bra_offset; k.ket_base = pd.class_off[kc];
  k.same_class = bc == kc;
  k.qclass = bc == 0 ? 0 : (bc == 1 ? 1 + kc : 3 + kc);
  k.chunk = tl.chunk;
  k.halves = tl.halves ? 1 : 0;
  k.maxp = pd.class_maxprim[bc];
  k.next = next;
  return k;
}

// The tests are made in float from float bounds (five roundings of 2^-24 at
// most and __fdividef's two units in the last place): thresholds and cuts are
// lowered by this much, so that no quartet and no primitive goes that the same
// test in double would keep.
constexpr float TEST_SLACK = 0.999999f;

constexpr int QUEUE = 64;  // a ring: up to 31 left over plus 32 new quartets
constexpr int MAXSLOT = 8;

// A queued quartet of this lane, as eval() gets it.
struct Queued {
  bool active;
  int ket, slot;  // ket pair within its class; slot of the staged bra
  int2 bra;       // {bra pair of the list, what stage() returned}
  float cut;
  bool one_bra;   // all active lanes share the bra
};

// A warp's walk over the tasks (see jk_split.cu): stage(bra, slot) stages a
// bra's records and returns a count, test(bra, ket, cut) the ring of a
// candidate or -1, eval(ring, quartet) evaluates 32 quartets.
template <int NRING, class StageFn, class TestFn, class EvalFn>
__device__ __forceinline__ void split_run(const SplitLists& L, int2 (*ring)[QUEUE], int2* slot_bra, StageFn stage,
                                          TestFn test, EvalFn eval) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int ntasks = L.ntasks_dev ? *L.ntasks_dev : L.ntasks;
  int qh[NRING] = {}, qn[NRING] = {}, slot = -1;
  unsigned long long used = 0;  // queued quartets per slot, one byte each
  int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int k = 0, k1 = 0, ib = 0;
  while (true) {
    int kind = -1;  // the ring to evaluate
#pragma unroll
    for (int r = 0; r < NRING; ++r)
      if (qn[r] >= 32) kind = r;
    if (kind < 0 && k >= k1 && t < ntasks) {
      const int next = (slot + 1) & (L.nslot - 1);
      if ((used >> (8 * next)) & 0xff) {  // its last bra still has queued quartets, the oldest of their rings
#pragma unroll
        for (int r = 0; r < NRING; ++r)
          if (qn[r] > 0 && (ring[r][qh[r]].x & (MAXSLOT - 1)) == next) kind = r;
      } else {  // next run
        slot = next;
        const int tg = L.task_begin + t;
        ib = find_bra(L.task_off, L.nbra, tg);
        k = __ldg(L.ket_lo + ib) + (tg - __ldg(L.task_off + ib)) * L.chunk;
        k1 = min(k + L.chunk, __ldg(L.ket_hi + ib));
        int more = 0;
        if (lane == 0) more = atomicAdd(L.next, 1);
        t = nw + __shfl_sync(0xffffffffu, more, 0);
        const int np = stage(ib, slot);
        if (lane == 0) slot_bra[slot] = make_int2(ib, np);
        __syncwarp();
      }
    }
    if (kind < 0 && k < k1) {
      float cut = 0.0f;
      const int ket = k + lane;
      const int to = ket < k1 ? test(ib, ket, cut) : -1;
      int added = 0;
#pragma unroll
      for (int r = 0; r < NRING; ++r) {
        const unsigned m = __ballot_sync(0xffffffffu, to == r);
        if (to == r)
          ring[r][(qh[r] + qn[r] + __popc(m & ((1u << lane) - 1u))) & (QUEUE - 1)] =
              make_int2(ket * MAXSLOT + slot, __float_as_int(cut));
        qn[r] += __popc(m);
        added += __popc(m);
      }
      used += (unsigned long long)added << (8 * slot);
      k += 32;
      __syncwarp();
      continue;
    }
    if (kind < 0) {  // the last quartets
#pragma unroll
      for (int r = 0; r < NRING; ++r)
        if (qn[r] > 0) kind = r;
      if (kind < 0) break;
    }
    // the ring's oldest 32 (or all there are): one quartet per lane
    const int have = NRING == 2 && kind == 1 ? qn[NRING - 1] : qn[0];
    const int head = NRING == 2 && kind == 1 ? qh[NRING - 1] : qh[0];
    const int n = min(have, 32);
    Queued q;
    q.active = lane < n;
    const int2 e = ring[kind][(head + (q.active ? lane : 0)) & (QUEUE - 1)];
    q.slot = e.x & (MAXSLOT - 1);
    q.ket = e.x / MAXSLOT;
    q.cut = __int_as_float(e.y);
#pragma unroll
    for (int r = 0; r < NRING; ++r)
      if (kind == r) {
        qh[r] = (qh[r] + n) & (QUEUE - 1);
        qn[r] -= n;
      }
    const int es0 = __shfl_sync(0xffffffffu, q.slot, 0);
    q.one_bra = __all_sync(0xffffffffu, !q.active || q.slot == es0);
    if (q.one_bra) used -= (unsigned long long)n << (8 * es0);
    else
      for (int x = 0; x < L.nslot; ++x)
        used -= (unsigned long long)__popc(__ballot_sync(0xffffffffu, q.active && q.slot == x)) << (8 * x);
    q.bra = slot_bra[q.slot];
    eval(kind, q);
    __syncwarp();  // the ring and slot entries read above may be overwritten
  }
}

// One unit of the bra and one ket primitive in the arithmetic type T (double
// or F2).
template <typename T> struct PrimSide {
  T P[3], k, p, o2p, A[3];  // k: the far prefactor or K; A: P-A or Q-C
};
template <bool KP, bool FAR>
__device__ __forceinline__ void load_ket(const KetTables& a, size_t sl, PrimSide<double>& k) {
  const double2 xy = a.xy[sl], zk = a.zk[sl];
  k.P[0] = xy.x; k.P[1] = xy.y; k.P[2] = zk.x; k.k = zk.y;
  if (!FAR) {
    const double2 pk = a.pk[sl];
    k.p = pk.x; k.k = pk.y;
  }
  k.A[0] = k.A[1] = k.A[2] = k.o2p = 0.0;
  if (KP) {
    const double2 pq = a.pq[sl], zo = a.zo[sl];
    k.A[0] = pq.x; k.A[1] = pq.y; k.A[2] = zo.x; k.o2p = zo.y;
  }
}
template <bool KP, bool FAR>
__device__ __forceinline__ void load_ket(const KetTables& a, size_t sl, PrimSide<F2>& k) {
  const float4 f = a.fp[sl];
  k.P[0] = F2(f.x); k.P[1] = F2(f.y); k.P[2] = F2(f.z); k.k = F2(f.w);
  if (!FAR) {
    const float2 pk = a.fk[sl];
    k.p = F2(pk.x); k.k = F2(pk.y);
  }
  k.A[0] = k.A[1] = k.A[2] = k.o2p = F2(0.0f);
  if (KP) {
    const float4 q = a.fq[sl];
    k.A[0] = F2(q.x); k.A[1] = F2(q.y); k.A[2] = F2(q.z); k.o2p = F2(q.w);
  }
}

template <typename T> struct Scalar { using R = T; };
template <> struct Scalar<F2> { using R = float; };

// A near primitive quartet (prim_setup of quartet.cuh with the short Boys table).
template <typename T, int L>
__device__ __forceinline__ void near_setup(const BoysRows<typename Scalar<T>::R>& tab, const T PQ[3],
                                           const PrimSide<T>& b, const PrimSide<T>& k, PrimGeo<T>& g) {
  const T rs = far_rsqrt(b.p + k.p);
  const T oz = rs * rs;
  const T tt = b.p * k.p * oz * pf_fma(PQ[0], PQ[0], pf_fma(PQ[1], PQ[1], PQ[2] * PQ[2]));
  const T pref = b.k * k.k * rs;
  T F[L + 1];
  boys_rows<L>(tab, tt, F);
#pragma unroll
  for (int m = 0; m <= L; ++m) g.I[m] = pref * F[m];
  if constexpr (L > 0) {
    const T pz = b.p * oz;
    g.nrp = k.p * oz * T(-1.0f);
    g.nrq = pz * T(-1.0f);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      g.WP[x] = g.nrp * PQ[x];
      g.WQ[x] = pz * PQ[x];
    }
    g.o2p = b.o2p;
    g.o2q = k.o2p;
    g.o2pq = T(0.5f) * oz;
  }
}

// Largest |D| of the exchange blocks of a quartet.
__device__ __forceinline__ float dmax_exchange(const float* __restrict__ dm, int ld, int a, int b, int c, int d) {
  return fmaxf(fmaxf(__ldg(dm + a * ld + c), __ldg(dm + a * ld + d)),
               fmaxf(__ldg(dm + b * ld + c), __ldg(dm + b * ld + d)));
}

}  // namespace pyfacc

// J/K digestion of long quartet lists in two halves: far quartets, all of
// whose primitive quartets are in the classical limit (far.cuh), and the rest.
//
// Both kernels walk the same tasks, a bra shell pair and a run of up to
// SPLIT_CHUNK_MAX ket pairs: a warp tests 32 candidates at a time
// (density-weighted Schwarz bound, distance), queues the survivors of its
// kernel's half in shared memory, and evaluates 32 whenever that many are
// queued, one contracted quartet per lane.  What is left of a run stays queued
// and is joined by the next runs', so lanes are full whatever the density
// screens out and however short the runs are, and all lanes take the same
// branches (the far half none of the Boys function's).  The far half keeps
// quartets that only J needs apart from those that K needs too: the exchange
// part of the digestion, four gathers and four atomics per quartet and
// density, is left out where Q_ab Q_cd max |D_ac, D_ad, D_bc, D_bd| stays below
// EXCHANGE_REL of the screening threshold.  One kernel with three rings did the candidate
// tests once, but needed the near half's registers throughout and was 5%
// slower.
//
// What bounds the kernels is the L1 data stage (wavefronts), then the FP64
// pipe: a 16-byte load that every lane takes from one address costs four
// wavefronts from global memory and two from shared memory, one of 32
// scattered records 14-20.  Hence the bras' primitive records are staged in
// shared memory, the kets are read from transposed records (KetTables), and
// the near half takes the Boys function from a conflict-free table
// (boys_rows.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "split.cuh"

namespace pyfacc {

namespace {

// What a far quartet that J needs may still add to K without being digested,
// relative to the screening threshold.  At 1 (the threshold of the quartets
// themselves) K of an SCF density moved by 4e-13 to 9e-13 of its norm against
// the kernels that digest everything, at 1e-3 by no more than the sums' own
// rounding (1e-15 to 9e-15, the same as without this test: C40H82, C100H202,
// gly30, C30H61).  FP64 build of C100H202: 11.08 ms at 1, 11.28 here, 11.54
// without; FP32 7.04, 7.23, 7.76.
constexpr float EXCHANGE_REL = 1e-3f;

struct SplitArgs {
  SplitLists l;
  JkArgs a;
  int prec;
};

// Staged bra records, in 16-byte vectors per unit: FP64 one primitive pair,
// FP32 two of them with their components interleaved (F2; an odd count is
// filled up with zero weight).
//   far:  {P, k}, with a p shell {P-A, 1/2p}
//   near: {P, p}, {K, 1/2p}, with a p shell {P-A}
// then |K| in float, for the primitive cut.
template <typename R, bool BP, bool FAR> struct Stage {
  static constexpr int VEC = FAR ? (BP ? 4 : 2) : (BP ? 5 : 3);
  static constexpr int UNIT = sizeof(R) == 8 ? 1 : 2;
  static __host__ __device__ constexpr int units(int n) { return (n + UNIT - 1) / UNIT; }
  static __host__ __device__ constexpr size_t bytes(int maxp) {
    return (size_t)units(maxp) * VEC * 16 + (size_t)(maxp + 3) / 4 * 16;
  }
  __device__ static __forceinline__ float* kab(unsigned char* st, int maxp) {
    return reinterpret_cast<float*>(st + (size_t)units(maxp) * VEC * 16);
  }
};

// Far bras on one atom have one product centre and are staged as their one
// equivalent primitive (KetTables row maxp).  Returns the staged count.
template <bool BP, bool FAR>
__device__ __forceinline__ int stage_bra(const SplitLists& a, int bra, const int4& bi0, double, unsigned char* st,
                                         int lane) {
  using S = Stage<double, BP, FAR>;
  const double4* br = a.prim + 3 * (size_t)bi0.z;
  double2* v = reinterpret_cast<double2*>(st);
  float* kab = S::kab(st, a.maxp);
  if (FAR) {
    const size_t m = (size_t)a.maxp * a.nbra_class + bra;
    const float km = a.bra.kabs[m];
    if (km > 0.0f) {
      if (lane == 0) {
        v[0] = a.bra.xy[m];
        v[1] = a.bra.zk[m];
        if (BP) {
          v[2] = a.bra.pq[m];
          v[3] = a.bra.zo[m];
        }
        kab[0] = km;
      }
      return 1;
    }
  }
  for (int i = lane; i < bi0.w; i += 32) {
    const double4 r0 = br[3 * i], r1 = br[3 * i + 1];
    double2* o = v + i * S::VEC;
    kab[i] = fabsf((float)r0.z);
    o[0] = make_double2(r1.x, r1.y);
    o[1] = make_double2(r1.z, FAR ? r1.w : r0.x);
    if (!FAR) o[2] = make_double2(r0.z, r0.y);
    if (BP) {
      const double4 r2 = br[3 * i + 2];
      o[S::VEC - 2] = make_double2(r2.x, r2.y);
      o[S::VEC - 1] = make_double2(r2.z, r2.w);
    }
  }
  return bi0.w;
}

template <bool BP, bool FAR>
__device__ __forceinline__ int stage_bra(const SplitLists& a, int bra, const int4& bi0, float, unsigned char* st,
                                         int lane) {
  using S = Stage<float, BP, FAR>;
  const float4* br = a.primf + 3 * (size_t)bi0.z;
  float* kab = S::kab(st, a.maxp);
  const size_t m = (size_t)a.maxp * a.nbra_class + bra;
  const float km = FAR ? a.bra.kabs[m] : 0.0f;
  const int np = km > 0.0f ? 1 : bi0.w;
  for (int i = lane; i < 2 * S::units(np); i += 32) {
    const int s = min(i, np - 1);
    const float w = i < np ? 1.0f : 0.0f;
    float4 r0 = make_float4(0.0f, 0.0f, km, 0.0f), r1, r2 = r0;
    if (km > 0.0f) {
      r1 = a.bra.fp[m];
      if (BP) r2 = a.bra.fq[m];
    } else {
      r0 = br[3 * s];
      r1 = br[3 * s + 1];
      if (BP) r2 = br[3 * s + 2];
    }
    float* o = reinterpret_cast<float*>(st) + (size_t)(i >> 1) * S::VEC * 4 + (i & 1);
    if (i < np) kab[i] = fabsf(r0.z);
    o[0] = r1.x; o[2] = r1.y; o[4] = r1.z;
    o[6] = FAR ? w * r1.w : r0.x;
    if (!FAR) {
      o[8] = w * r0.z;
      o[10] = r0.y;
    }
    if (BP) {
      float* q = o + (S::VEC - 2) * 4;
      q[0] = r2.x; q[2] = r2.y; q[4] = r2.z; q[6] = r2.w;
    }
  }
  return np;
}

template <bool BP, bool FAR>
__device__ __forceinline__ void load_unit(const unsigned char* st, int i, PrimSide<double>& b) {
  using S = Stage<double, BP, FAR>;
  const double2* v = reinterpret_cast<const double2*>(st) + i * S::VEC;
  const double2 a0 = v[0], a1 = v[1];
  b.P[0] = a0.x; b.P[1] = a0.y; b.P[2] = a1.x;
  b.o2p = 0.0;
  if (FAR) {
    b.k = a1.y;
  } else {
    const double2 a2 = v[2];
    b.p = a1.y; b.k = a2.x; b.o2p = a2.y;
  }
  b.A[0] = b.A[1] = b.A[2] = 0.0;
  if (BP) {
    const double2 c0 = v[S::VEC - 2], c1 = v[S::VEC - 1];
    b.A[0] = c0.x; b.A[1] = c0.y; b.A[2] = c1.x; b.o2p = c1.y;
  }
}
template <bool BP, bool FAR>
__device__ __forceinline__ void load_unit(const unsigned char* st, int i, PrimSide<F2>& b) {
  using S = Stage<float, BP, FAR>;
  const float4* v = reinterpret_cast<const float4*>(st) + i * S::VEC;
  const float4 a0 = v[0], a1 = v[1];
  b.P[0] = F2(a0.x, a0.y); b.P[1] = F2(a0.z, a0.w); b.P[2] = F2(a1.x, a1.y);
  b.o2p = F2(0.0f);
  if (FAR) {
    b.k = F2(a1.z, a1.w);
  } else {
    const float4 a2 = v[2];
    b.p = F2(a1.z, a1.w); b.k = F2(a2.x, a2.y); b.o2p = F2(a2.z, a2.w);
  }
  b.A[0] = b.A[1] = b.A[2] = F2(0.0f);
  if (BP) {
    const float4 c0 = v[S::VEC - 2], c1 = v[S::VEC - 1];
    b.A[0] = F2(c0.x, c0.y); b.A[1] = F2(c0.z, c0.w); b.A[2] = F2(c1.x, c1.y); b.o2p = F2(c1.z, c1.w);
  }
}
template <typename T, int LA, int LB, int LC, int LD, bool FAR>
__device__ __forceinline__ void add_prim(const BoysRows<typename Scalar<T>::R>& tab, const PrimSide<T>& b,
                                         const PrimSide<T>& k, T* __restrict__ acc) {
  using C = EriClass<T, LA, LB, LC, LD>;
  T PQ[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) PQ[x] = b.P[x] + k.P[x] * T(-1.0f);
  PrimGeo<T> g;
  if constexpr (FAR) far_setup<T, C::L>(PQ, b.k * k.k, b.o2p, k.o2p, g);
  else near_setup<T, C::L>(tab, PQ, b, k, g);
  C::vrr(g.I, b.A, g.WP, k.A, g.WQ, g.o2p, g.nrp, g.o2q, g.nrq, g.o2pq, acc);
}

__device__ __forceinline__ void sum_acc(const double* a, int i, double* o) { o[i] = a[i]; }
__device__ __forceinline__ void sum_acc(const F2* a, int i, float* o) { o[i] = a[i].v.x + a[i].v.y; }

// Contracted (ab|cd) of one lane; returns the primitive quartets summed.  The
// primitive pairs are sorted by |K|: the bra prefix that passes the cut only
// shrinks from one ket primitive to the next.  Light far classes take two ket
// primitives per pass over the bra, which halves the bra's loads.
template <typename R, int LA, int LB, int LC, int LD, bool FAR>
__device__ __forceinline__ int quartet(const SplitLists& a, const BoysRows<R>& tab, unsigned char* st, int np, int ket,
                                       int nk, const double4& bgeo, const double4& kgeo, float cut,
                                       R* __restrict__ out) {
  constexpr bool BP = LA + LB > 0, KP = LC + LD > 0;
  using S = Stage<R, BP, FAR>;
  using T = typename std::conditional<sizeof(R) == 8, double, F2>::type;
  using C1 = EriClass<R, LA, LB, LC, LD>;
  constexpr bool TWO = FAR && sizeof(R) == 8 && C1::L <= 1;
  const float* kab = S::kab(st, a.maxp);
  T acc[C1::NACC];
#pragma unroll
  for (int i = 0; i < C1::NACC; ++i) acc[i] = T(0.0f);
  int n = np, nprim = 0, kq = 0;
  if (FAR && a.ket.kabs[(size_t)a.ketmaxp * a.nket + ket] > 0.0f) {  // a ket on one atom: its equivalent primitive
    kq = a.ketmaxp;
    nk = kq + 1;
  }
  for (; kq < nk; ++kq) {
    size_t sl = (size_t)kq * a.nket + ket;
    float kcd = a.ket.kabs[sl];
    PrimSide<T> k;
    load_ket<KP, FAR>(a.ket, sl, k);
    while (n > 0 && kab[n - 1] * kcd < cut) --n;
    if (n == 0) break;
    nprim += n;
    if constexpr (TWO) {
      const int n0 = n;
      int i = 0;
      if (++kq < nk) {
        sl += a.nket;
        kcd = a.ket.kabs[sl];
        PrimSide<T> k2;
        load_ket<KP, FAR>(a.ket, sl, k2);
        while (n > 0 && kab[n - 1] * kcd < cut) --n;
        nprim += n;
        for (; i < n; ++i) {
          PrimSide<T> b;
          load_unit<BP, FAR>(st, i, b);
          add_prim<T, LA, LB, LC, LD, FAR>(tab, b, k, acc);
          add_prim<T, LA, LB, LC, LD, FAR>(tab, b, k2, acc);
        }
      }
#pragma unroll 1
      for (; i < n0; ++i) {
        PrimSide<T> b;
        load_unit<BP, FAR>(st, i, b);
        add_prim<T, LA, LB, LC, LD, FAR>(tab, b, k, acc);
      }
    } else {
      const int nu = S::units(n);
#pragma unroll 1
      for (int i = 0; i < nu; ++i) {
        PrimSide<T> b;
        load_unit<BP, FAR>(st, i, b);
        add_prim<T, LA, LB, LC, LD, FAR>(tab, b, k, acc);
      }
    }
  }
  R accs[C1::NACC];
#pragma unroll
  for (int i = 0; i < C1::NACC; ++i) sum_acc(acc, i, accs);
  const R AB[3] = {(R)bgeo.x, (R)bgeo.y, (R)bgeo.z}, CD[3] = {(R)kgeo.x, (R)kgeo.y, (R)kgeo.z};
  C1::hrr(accs, AB, CD, out);
  return nprim;
}

// Resident blocks per SM that the registers are held to (8 / 6 / 5 instead of
// 7 / 5 / 4 for L = 0 / 1 / 2: FP32 builds -4%, FP64 the same despite spills).
__host__ __device__ constexpr int min_blocks(int L) {
  return L == 0 ? 8 : (L == 1 ? 6 : (L == 2 ? 5 : 3));
}

template <typename R, int LA, int LB, int LC, int LD, int NK, bool FAR>
__global__ void __launch_bounds__(128, min_blocks(LA + LB + LC + LD)) jk_split_kernel(const SplitArgs args) {
  using C = EriClass<R, LA, LB, LC, LD>;
  using S = Stage<R, (LA + LB > 0), FAR>;
  constexpr int NRING = FAR ? 2 : 1;  // far: 0 only J, 1 J and K
  constexpr int NA = NC<LA>::v, NB = NC<LB>::v, NCc = NC<LC>::v, ND = NC<LD>::v;
  extern __shared__ __align__(16) unsigned char split_smem[];
  __shared__ int2 queue[4][NRING][QUEUE];  // {ket * MAXSLOT + slot, primitive cut}
  __shared__ int2 slot_bra[4][MAXSLOT];    // {bra, staged primitive pairs}
  __shared__ unsigned count[4][NRING];     // quartets evaluated
  __shared__ typename std::conditional<FAR, int, BoysRows<R>>::type tab_smem;
  const BoysRows<R>& tab = reinterpret_cast<const BoysRows<R>&>(tab_smem);  // near half only
  if constexpr (!FAR) {
    const unsigned* src = static_cast<const unsigned*>(args.l.boys);
    unsigned* dst = reinterpret_cast<unsigned*>(&tab_smem);
    for (int i = threadIdx.x; i < (int)(sizeof(BoysRows<R>) / 4); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const SplitLists& L = args.l;
  const JkArgs& A = args.a;
  const size_t slot_bytes = S::bytes(L.maxp);
  unsigned char* st = split_smem + (size_t)wib * L.nslot * slot_bytes;
  if (lane < NRING) count[wib][lane] = 0;
  __syncwarp();
  unsigned nprim = 0;
  auto stage = [&](int ib, int slot) {
    return stage_bra<(LA + LB > 0), FAR>(L, L.bra_off + ib, L.info0[L.bra_base + ib], (R)0, st + slot * slot_bytes,
                                         lane);
  };
  auto test = [&](int ib, int ket, float& cut) {
    const int bp = L.bra_base + ib, kp = L.ket_base + ket;
    const float4 bc = L.test[bp], bt = L.test2[bp], kc = L.test[kp], kt = L.test2[kp];
    if ((FAR || L.halves) &&
        far_pair(bc, far_extent<R, C::L>(bc.w, bt.x), kc, far_extent<R, C::L>(kc.w, kt.x)) != FAR)
      return -1;
    int to = NRING - 1;
    if (A.dmax) {
      const float* dmx = A.dmax + L.info2[bp].w;
      const int sa = __float_as_int(bt.z), sb = __float_as_int(bt.w), sc = __float_as_int(kt.z),
                sd = __float_as_int(kt.w);
      const float dk = dmax_exchange(dmx, A.ns_ld, sa, sb, sc, sd);
      const float dm = fmaxf(2.0f * fmaxf(__ldg(dmx + sa * A.ns_ld + sb), __ldg(dmx + sc * A.ns_ld + sd)), dk);
      const float qq = bt.y * kt.y;
      const float thr = TEST_SLACK * (float)A.thresh;
      if (!(qq * dm >= thr)) return -1;
      if (FAR && !(qq * dk >= EXCHANGE_REL * thr)) to = 0;
      cut = TEST_SLACK * __fdividef((float)A.prim_thresh, fmaxf(dm, 1e-30f));
    }
    return to;
  };
  auto eval = [&](int kind, const Queued& q) {
    const int bp = L.bra_base + q.bra.x, kp = L.ket_base + q.ket;
    const int4 bi0 = L.info0[bp], ki0 = L.info0[kp], bi2 = L.info2[bp];
    const int mo = bi2.x, ld = bi2.y, ma = bi0.x, mb = bi0.y, mc = ki0.x, md = ki0.y;
    if (A.stats) {  // per warp and ring (a register per lane for it spilled)
      const unsigned m = __ballot_sync(0xffffffffu, q.active);
      if (lane == 0) count[wib][kind] += __popc(m);
    }
    double jab[NA * NB];
#pragma unroll
    for (int i = 0; i < NA * NB; ++i) jab[i] = 0.0;
    if (q.active) {
      R out[C::NOUT];
      nprim += quartet<R, LA, LB, LC, LD, FAR>(L, tab, st + q.slot * slot_bytes, q.bra.y, q.ket, ki0.w, L.geom[bp],
                                               L.geom[kp], q.cut, out);
      double fac = 1.0;
      const float4 bt = L.test2[bp], kt = L.test2[kp];
      if (__float_as_int(bt.z) == __float_as_int(bt.w)) fac *= 0.5;
      if (__float_as_int(kt.z) == __float_as_int(kt.w)) fac *= 0.5;
      if (L.same_class && bp == kp) fac *= 0.5;
      // ---- Coulomb
      double Dab[NA * NB], jcd[NCc * ND];
#pragma unroll
      for (int i = 0; i < NA * NB; ++i) Dab[i] = __ldg(A.Dj + mo + (ma + i / NB) * ld + mb + i % NB);
#pragma unroll
      for (int i = 0; i < NCc * ND; ++i) jcd[i] = 0.0;
#pragma unroll
      for (int c = 0; c < NCc; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const double Dcd = __ldg(A.Dj + mo + (mc + c) * ld + md + d);
#pragma unroll
          for (int i = 0; i < NA * NB; ++i) {
            const double v = fac * (double)out[(i * NCc + c) * ND + d];
            jab[i] += v * Dcd;
            jcd[c * ND + d] += v * Dab[i];
          }
        }
#pragma unroll
      for (int c = 0; c < NCc; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) atomicAdd(A.J + mo + (mc + c) * ld + md + d, 2.0 * jcd[c * ND + d]);
      // ---- exchange, one or two densities
      if (!FAR || kind == 1) {
#pragma unroll
        for (int kd = 0; kd < NK; ++kd) {
          const double* Dk = ((kd == 0) ? A.Dk0 : A.Dk1) + mo;
          double* Kk = ((kd == 0) ? A.K0 : A.K1) + mo;
          double kac[NA * NCc], kad[NA * ND], kbc[NB * NCc], kbd[NB * ND];
          double Dbd[NB * ND], Dbc[NB * NCc], Dad[NA * ND], Dac[NA * NCc];
#pragma unroll
          for (int a = 0; a < NA; ++a) {
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              Dad[a * ND + d] = __ldg(Dk + (ma + a) * ld + md + d);
              kad[a * ND + d] = 0.0;
            }
#pragma unroll
            for (int c = 0; c < NCc; ++c) {
              Dac[a * NCc + c] = __ldg(Dk + (ma + a) * ld + mc + c);
              kac[a * NCc + c] = 0.0;
            }
          }
#pragma unroll
          for (int b = 0; b < NB; ++b) {
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              Dbd[b * ND + d] = __ldg(Dk + (mb + b) * ld + md + d);
              kbd[b * ND + d] = 0.0;
            }
#pragma unroll
            for (int c = 0; c < NCc; ++c) {
              Dbc[b * NCc + c] = __ldg(Dk + (mb + b) * ld + mc + c);
              kbc[b * NCc + c] = 0.0;
            }
          }
#pragma unroll
          for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
              for (int c = 0; c < NCc; ++c)
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                  const double v = fac * (double)out[((a * NB + b) * NCc + c) * ND + d];
                  kac[a * NCc + c] += v * Dbd[b * ND + d];
                  kad[a * ND + d] += v * Dbc[b * NCc + c];
                  kbc[b * NCc + c] += v * Dad[a * ND + d];
                  kbd[b * ND + d] += v * Dac[a * NCc + c];
                }
#pragma unroll
          for (int a = 0; a < NA; ++a) {
#pragma unroll
            for (int c = 0; c < NCc; ++c) atomicAdd(Kk + (ma + a) * ld + mc + c, kac[a * NCc + c]);
#pragma unroll
            for (int d = 0; d < ND; ++d) atomicAdd(Kk + (ma + a) * ld + md + d, kad[a * ND + d]);
          }
#pragma unroll
          for (int b = 0; b < NB; ++b) {
#pragma unroll
            for (int c = 0; c < NCc; ++c) atomicAdd(Kk + (mb + b) * ld + mc + c, kbc[b * NCc + c]);
#pragma unroll
            for (int d = 0; d < ND; ++d) atomicAdd(Kk + (mb + b) * ld + md + d, kbd[b * ND + d]);
          }
        }
      }
    }
    // J_ab: one atomic per warp while all lanes share the bra
    if (q.one_bra) {
#pragma unroll
      for (int i = 0; i < NA * NB; ++i) {
        const double s = warp_sum(jab[i]);
        if (lane == 0) atomicAdd(A.J + mo + (ma + i / NB) * ld + mb + i % NB, 2.0 * s);
      }
    } else if (q.active) {
#pragma unroll
      for (int i = 0; i < NA * NB; ++i) atomicAdd(A.J + mo + (ma + i / NB) * ld + mb + i % NB, 2.0 * jab[i]);
    }
  };
  split_run<NRING>(L, queue[wib], slot_bra[wib], stage, test, eval);
  if (A.stats) {  // contracted and evaluated primitive quartets
    unsigned long long p = nprim;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
    const unsigned long long nj = count[wib][0], nq = NRING == 2 ? nj + count[wib][NRING - 1] : nj;
    if (lane == 0 && nq) {
      atomicAdd(A.stats + args.prec * NQCLASS + L.qclass, nq);
      atomicAdd(A.stats + (2 + args.prec) * NQCLASS + L.qclass, p);
      if (FAR) {
        atomicAdd(A.stats + JK_STATS_FAR + args.prec * NQCLASS + L.qclass, p);
        atomicAdd(A.stats + JK_STATS_J_ONLY + args.prec * NQCLASS + L.qclass, nj);
      }
    }
  }
}

// Shared memory for the staged bras of a block: eight runs per warp, fewer for
// deep contractions (STO-6G: 36 primitive pairs).
constexpr size_t STAGE_MAX_BYTES = 24 * 1024;

template <typename R, int LA, int LB, int LC, int LD, int NK, bool FAR>
void launch_one(int blocks, cudaStream_t s, SplitArgs k) {
  const size_t b = Stage<R, (LA + LB > 0), FAR>::bytes(k.l.maxp);
  k.l.nslot = MAXSLOT;
  while (k.l.nslot > 2 && 4 * k.l.nslot * b > STAGE_MAX_BYTES) k.l.nslot /= 2;
  const size_t smem = 4 * k.l.nslot * b;
  if (smem > 32 * 1024)
    allow_smem(jk_split_kernel<R, LA, LB, LC, LD, NK, FAR>,
               std::max(STAGE_MAX_BYTES, 4 * 2 * Stage<R, (LA + LB > 0), FAR>::bytes(SPLIT_MAXPRIM)));
  jk_split_kernel<R, LA, LB, LC, LD, NK, FAR><<<blocks, 128, smem, s>>>(k);
  PF_CUDA(cudaGetLastError());
  count_split_launch(FAR);
}

template <typename R, int LA, int LB, int LC, int LD>
void launch_halves(int nk, int blocks, cudaStream_t s_far, cudaStream_t s_near, SplitArgs k) {
  if (nk == 1) {
    launch_one<R, LA, LB, LC, LD, 1, false>(blocks, s_near, k);
    ++k.l.next;
    if (k.l.halves) launch_one<R, LA, LB, LC, LD, 1, true>(blocks, s_far, k);
  } else {
    launch_one<R, LA, LB, LC, LD, 2, false>(blocks, s_near, k);
    ++k.l.next;
    if (k.l.halves) launch_one<R, LA, LB, LC, LD, 2, true>(blocks, s_far, k);
  }
}

template <typename R>
void dispatch(int qc, int nk, int blocks, cudaStream_t s_far, cudaStream_t s_near, const SplitArgs& k) {
  switch (qc) {
    case 0: launch_halves<R, 0, 0, 0, 0>(nk, blocks, s_far, s_near, k); break;
    case 1: launch_halves<R, 1, 0, 0, 0>(nk, blocks, s_far, s_near, k); break;
    case 2: launch_halves<R, 1, 0, 1, 0>(nk, blocks, s_far, s_near, k); break;
    case 3: launch_halves<R, 1, 1, 0, 0>(nk, blocks, s_far, s_near, k); break;
    default: launch_halves<R, 1, 1, 1, 0>(nk, blocks, s_far, s_near, k); break;
  }
}

}  // namespace

// Kets per run of a list that the split kernels take, 0 for one they do not.
// They pay for their second pass over the candidates with the far quartets:
// with 3e5 of them per class and more the whole build gains (C20H42 (ss|ss):
// 4e5, FP64 build 1.00 -> 0.87 ms; C40H82 2.60 -> 2.47 ms with (pp|ss) and
// (pp|ps), 3e5 and 5e5, too), while a cluster of 16 waters, 5e5 quartets of
// which next to none are far, loses (0.46 -> 0.63 ms).  far_share is the share
// of atom pairs beyond FAR_DISTANCE.
// FP64 lists of the deepest contractions need twice as many: their few runs
// last too long to share evenly (STO-6G, FP64 build of C16H34 5.2 ms undivided,
// 5.9 divided, C18H38 6.6 and 7.2, C20H42 8.2 and 8.0; in FP32 2.75 and 2.49,
// 3.54 and 3.02, 4.36 and 3.41; STO-4G C18H38 FP64 1.74 and 1.67).
int split_chunk(long long nquartets, double far_share, int prim_quartets, bool fp32, int num_sms) {
  const double line = !fp32 && prim_quartets > SPLIT_DEEP ? 2.0 * SPLIT_MIN_FAR : SPLIT_MIN_FAR;
  return (double)nquartets * far_share < line ? 0 : split_run(nquartets, prim_quartets, num_sms);
}

// Runs as long as leave SPLIT_RUNS_PER_SM per SM, more for deep contractions,
// whose quartets take longer.
int split_run(long long nquartets, int prim_quartets, int num_sms) {
  const long long runs = (long long)num_sms * SPLIT_RUNS_PER_SM * std::min(4, std::max(1, prim_quartets / 81));
  int c = 32;
  while (c < SPLIT_CHUNK_MAX && nquartets / (2 * c) >= runs) c *= 2;
  return c;
}

// (pp|pp) keeps the undivided kernel: few quartets, and its time is the
// recursion's, not the Boys function's.
bool split_class(const PairData& pd, int bc, int kc) {
  return bc < NCLASS && !(bc == 2 && kc == 2) && pd.class_maxprim[bc] <= SPLIT_MAXPRIM;
}

bool jk_splits(const PairData& pd, const TaskList& tl) { return pd.kt.xy && tl.chunk > 0; }

void launch_jk_split(const PairData& pd, const TaskList& tl, int bc, int kc, bool fp32, int nk, const JkArgs& a,
                     int num_sms, int* next, cudaStream_t s_far, cudaStream_t s_near) {
  if (tl.ntasks_c <= 0) return;
  if (fp32 && !pd.primf) throw Error(PYFACC_ERR_INVALID, "FP32 quartets need float primitive records");
  SplitArgs k{};
  k.l = split_lists(pd, tl, bc, kc, next);
  k.l.boys = boys_rows_table(fp32, class_flops(k.l.qclass).L);
  k.a = a;
  k.prec = fp32 ? 1 : 0;
  // resident warps only; the tasks beyond their first go to whichever is free
  const int per_sm = min_blocks(class_flops(k.l.qclass).L);
  const int blocks = (int)std::max(1LL, std::min((tl.ntasks_c + 3LL) / 4, (long long)num_sms * per_sm));
  if (fp32) dispatch<float>(k.l.qclass, nk, blocks, s_far, s_near, k);
  else dispatch<double>(k.l.qclass, nk, blocks, s_far, s_near, k);
}

}  // namespace pyfacc

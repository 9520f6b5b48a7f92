// Gradient of one primitive quartet of s and p shells contracted with its
// density products, in Hermite Gaussians (McMurchie and Davidson 1978).
//
// The bra product p_i p_j about P is the Hermite series
//   (PA_i PB_j + d_ij h) + h PB_j L_i + h PA_i L_j + h^2 L_ij,   h = 1/2p,
// so the energy sum Gamma_ijkl (ij|kl) is a sum of Hermite densities H_T, 35
// for (pp|pp), times the Hermite integrals R_T of P - Q, its derivative along P
// the same sum with R_(T+x), and the derivatives along A - B at fixed P the
// partial sums behind PA, PB and the prefactor.  A = P + (b/p) X, B = P - (a/p) X
// with X = A - B gives the centres'.  The Obara-Saika routines that these
// replace built the raised and lowered integrals of every centre: 9480 flops a
// primitive quartet for (pp|pp), here 3350, 4848 for (pp|ps), here 1000, or 66
// and 69 accumulators a lane for (pp|ss) and (ps|ps), which filled the register
// file.  The kernels are bound by the FP64 pipe and by the registers: FP64
// gradient of C40H82 8.7 -> 5.9 ms, gly30 52 -> 26 ms, C30H61 (STO-6G, UHF) 55
// -> 36 ms, FP32 (pp|pp) of gly30 5.3 -> 1.2 ms, (pp|ps) 4.9 -> 2.6 ms.  In the
// undivided FP32 kernels (ps|ss), (ps|ps), (pp|ss) wait for loads either way
// (C100H202: 10.5 / 4.2 / 1.8 ms, with this 10.5 / 4.1 / 1.6) and keep the
// contracted accumulators.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "eri_classes.cuh"

namespace pyfacc {

// Index of the Hermite Gaussian (t, u, v): by order, then by falling t, u.
constexpr int herm_index(int t, int u, int v) {
  const int n = t + u + v;
  return n * (n + 1) * (n + 2) / 6 + (n - t) * (n - t + 1) / 2 + v;
}
constexpr int herm_count(int order) { return (order + 1) * (order + 2) * (order + 3) / 6; }
struct Herm {
  int t, u, v;
  constexpr int operator[](int x) const { return x == 0 ? t : (x == 1 ? u : v); }
};
constexpr Herm herm_of(int index) {
  int n = 0;
  while (herm_count(n) <= index) ++n;
  int r = index - n * (n + 1) * (n + 2) / 6, a = 0;  // a = n - t
  while ((a + 1) * (a + 2) / 2 <= r) ++a;
  const int v = r - a * (a + 1) / 2;
  return Herm{n - a, a - v, v};
}
// Index of h raised by one along x (x < 0: h itself).
constexpr int herm_add(int h, int x) {
  const Herm a = herm_of(h);
  return herm_index(a.t + (x == 0), a.u + (x == 1), a.v + (x == 2));
}

template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// One level of the Hermite integrals, m + 1 -> m, for orders up to n:
// R^(m)_(T+x) = PQ_x R^(m+1)_T + T_x R^(m+1)_(T-x), in place from the highest
// order down.  use(h, R_h) sees every result; those beyond the KEEP first are
// not stored.
template <typename T, int n, int KEEP, class Use>
__device__ __forceinline__ void herm_level(const T* PQ, T r0, T* r, Use&& use) {
  static_for<herm_count(n) - 1>([&](auto rev) {
    constexpr int h = herm_count(n) - 1 - decltype(rev)::value;
    constexpr Herm a = herm_of(h);
    // along an axis with exponent 1 there is no second term
    constexpr int x = a.t == 1 ? 0 : (a.u == 1 ? 1 : (a.v == 1 ? 2 : (a.t > 1 ? 0 : (a.u > 1 ? 1 : 2))));
    constexpr int e = a[x];
    constexpr int h1 = herm_index(a.t - (x == 0), a.u - (x == 1), a.v - (x == 2));
    T v = PQ[x] * r[h1];
    if constexpr (e > 1) {
      constexpr int h2 = herm_index(a.t - 2 * (x == 0), a.u - 2 * (x == 1), a.v - 2 * (x == 2));
      if constexpr (e == 2) v = pf_fma(PQ[x], r[h1], r[h2]);
      else v = pf_fma(PQ[x], r[h1], T((float)(e - 1)) * r[h2]);
    }
    if constexpr (h < KEEP) r[h] = v;
    use(std::integral_constant<int, h>{}, v);
  });
  r[0] = r0;
  use(std::integral_constant<int, 0>{}, r0);
}

// One side of a primitive quartet.
template <typename T> struct MdSide {
  T A[3], B[3];   // P - first centre, P - second centre
  T h;            // 1/2p
  T fa, fb;       // a/p, b/p
  T mu2;          // 2ab/p
};
template <typename T>
__device__ __forceinline__ void md_side(const T* PA, const T* AB, T h, T ta, T tb, MdSide<T>& s) {
  s.h = h;
  s.fa = ta * h;
  s.fb = tb * h;
  s.mu2 = ta * s.fb;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    s.A[x] = PA[x];
    s.B[x] = PA[x] + AB[x];
  }
}

// BL, KL: the bra and the ket are (ss), (ps) or (pp).
// I[m], m = 0 .. L + 1, are the Boys values with prefactor and scale = -2 rho
// (in the far limit, where I carries rho^m, -2).  gam(i, j, k, l): the density
// products, indices of an s shell 0.  Adds dE/dA, dE/dB, dE/dC to g.
template <typename T, int BL, int KL, class Gam>
__device__ __forceinline__ void md_gradient(const T* I, T scale, const T* PQ, const MdSide<T>& b, const MdSide<T>& k,
                                            Gam&& gam, T* g) {
  constexpr bool BB = BL == 2;
  constexpr int L = BL + KL, NB = BB ? 3 : 1, NC = KL > 0 ? 3 : 1, ND = KL == 2 ? 3 : 1, NHB = herm_count(BL);
  const T zero = T(0.0f), mone = T(-1.0f);
  const T h2 = b.h * b.h, kh = k.h * mone, kh2 = k.h * k.h;
  // ket coefficients of L_0, L_c, L_d (L_cd: kh2); the signs are those of d/dQ
  auto ket = [&](int c, int d, T& c0, T& cc, T& cd) {
    c0 = T(1.0f);
    cc = cd = zero;
    if constexpr (KL == 2) {
      c0 = pf_fma(k.A[c], k.B[d], c == d ? k.h : zero);
      cc = kh * k.B[d];
      cd = kh * k.A[c];
    } else if constexpr (KL == 1) {
      c0 = k.A[c];
      cc = kh;
    }
  };
  // ---- Hermite densities
  T H[herm_count(L)];
#pragma unroll
  for (int i = 0; i < herm_count(L); ++i) H[i] = zero;
  static_for<NC * ND>([&](auto cd) {
    constexpr int c = decltype(cd)::value / ND, d = decltype(cd)::value % ND;
    T h[NHB];
    if constexpr (BB) {
      T G[3][3], s[3], r[3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) G[i][j] = gam(i, j, c, d);
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        s[x] = pf_fma(G[0][x], b.A[0], pf_fma(G[1][x], b.A[1], G[2][x] * b.A[2]));
        r[x] = pf_fma(G[x][0], b.B[0], pf_fma(G[x][1], b.B[1], G[x][2] * b.B[2]));
      }
      h[0] = pf_fma(s[0], b.B[0], pf_fma(s[1], b.B[1], pf_fma(s[2], b.B[2], b.h * (G[0][0] + G[1][1] + G[2][2]))));
#pragma unroll
      for (int x = 0; x < 3; ++x) h[1 + x] = b.h * (s[x] + r[x]);
      h[herm_index(2, 0, 0)] = h2 * G[0][0];
      h[herm_index(0, 2, 0)] = h2 * G[1][1];
      h[herm_index(0, 0, 2)] = h2 * G[2][2];
      h[herm_index(1, 1, 0)] = h2 * (G[0][1] + G[1][0]);
      h[herm_index(1, 0, 1)] = h2 * (G[0][2] + G[2][0]);
      h[herm_index(0, 1, 1)] = h2 * (G[1][2] + G[2][1]);
    } else if constexpr (BL == 0) {
      h[0] = gam(0, 0, c, d);
    } else {
      const T G[3] = {gam(0, 0, c, d), gam(1, 0, c, d), gam(2, 0, c, d)};
      h[0] = pf_fma(G[0], b.A[0], pf_fma(G[1], b.A[1], G[2] * b.A[2]));
#pragma unroll
      for (int x = 0; x < 3; ++x) h[1 + x] = b.h * G[x];
    }
    T c0, cc, c1;
    ket(c, d, c0, cc, c1);
    static_for<NHB>([&](auto hh) {
      constexpr int i = decltype(hh)::value;
      if constexpr (KL == 0) {
        H[i] = h[i];
      } else {
        constexpr int ic = herm_add(i, c);
        H[i] = pf_fma(c0, h[i], H[i]);
        H[ic] = pf_fma(cc, h[i], H[ic]);
        if constexpr (KL == 2) {
          constexpr int id = herm_add(i, d), icd = herm_add(ic, d);
          H[id] = pf_fma(c1, h[i], H[id]);
          H[icd] = pf_fma(kh2, h[i], H[icd]);
        }
      }
    });
  });
  // ---- Hermite integrals, the energy and its derivative along P.  The last
  // level is used as it arises: its highest order is needed here alone.
  T R[herm_count(L)], E = zero, dP[3] = {zero, zero, zero};
  {
    T base[L + 2], f = scale;
    base[0] = I[0];
#pragma unroll
    for (int m = 1; m <= L + 1; ++m) {
      base[m] = I[m] * f;
      f = f * scale;
    }
    R[0] = base[L + 1];
    static_for<L>([&](auto lev) {
      constexpr int n = decltype(lev)::value + 1;
      herm_level<T, n, herm_count(L)>(PQ, base[L + 1 - n], R, [](auto, T) {});
    });
    herm_level<T, L + 1, herm_count(L)>(PQ, base[0], R, [&](auto hh, T v) {
      constexpr int h = decltype(hh)::value;
      constexpr Herm a = herm_of(h);
      if constexpr (a.t > 0) dP[0] = pf_fma(H[herm_index(a.t - 1, a.u, a.v)], v, dP[0]);
      if constexpr (a.u > 0) dP[1] = pf_fma(H[herm_index(a.t, a.u - 1, a.v)], v, dP[1]);
      if constexpr (a.v > 0) dP[2] = pf_fma(H[herm_index(a.t, a.u, a.v - 1)], v, dP[2]);
      if constexpr (h < herm_count(L)) E = pf_fma(H[h], v, E);
    });
  }
  // ---- along A - B at fixed P: d/dPA_i = sum_j Gamma_ij (PB_j V_0 + h V_j),
  // d/dPB_j = sum_i Gamma_ij (PA_i V_0 + h V_i) with V the ket's potentials
  T dX[3], dY[3];
  const T me = mone * E;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    dX[x] = b.mu2 * (b.B[x] + mone * b.A[x]) * me;
    dY[x] = k.mu2 * (k.B[x] + mone * k.A[x]) * me;
  }
  const T mfb = mone * b.fb, mkb = mone * k.fb;
  static_for<(BL > 0 ? NC * ND : 0)>([&](auto cd) {
    constexpr int c = decltype(cd)::value / ND, d = decltype(cd)::value % ND;
    T c0, cc, c1, V[4];
    ket(c, d, c0, cc, c1);
    static_for<(BB ? 4 : 1)>([&](auto hh) {
      constexpr int i = decltype(hh)::value;
      if constexpr (KL == 0) {
        V[i] = R[i];
      } else {
        constexpr int ic = herm_add(i, c);
        V[i] = pf_fma(c0, R[i], cc * R[ic]);
        if constexpr (KL == 2) {
          constexpr int id = herm_add(i, d), icd = herm_add(ic, d);
          V[i] = pf_fma(c1, R[id], pf_fma(kh2, R[icd], V[i]));
        }
      }
    });
    if constexpr (BB) {
      T U[3], W[3];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const T hv = b.h * V[1 + x];
        U[x] = mfb * pf_fma(b.B[x], V[0], hv);
        W[x] = b.fa * pf_fma(b.A[x], V[0], hv);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const T G = gam(i, j, c, d);
          dX[i] = pf_fma(G, U[j], dX[i]);
          dX[j] = pf_fma(G, W[i], dX[j]);
        }
    } else {
      const T u = mfb * V[0];
#pragma unroll
      for (int i = 0; i < 3; ++i) dX[i] = pf_fma(gam(i, 0, c, d), u, dX[i]);
    }
  });
  // ---- along C - D at fixed Q, from the bra's potentials
  if constexpr (KL > 0)
    static_for<3 * NB>([&](auto ij) {
      constexpr int i = decltype(ij)::value / NB, j = decltype(ij)::value % NB;
      T V[4];
      if constexpr (BB) {
        const T b0 = pf_fma(b.A[i], b.B[j], i == j ? b.h : zero), bi = b.h * b.B[j], bj = b.h * b.A[i];
        static_for<(KL == 2 ? 4 : 1)>([&](auto hh) {
          constexpr int m = decltype(hh)::value, mi = herm_add(m, i), mj = herm_add(m, j), mij = herm_add(mi, j);
          V[m] = pf_fma(b0, R[m], pf_fma(bi, R[mi], pf_fma(bj, R[mj], h2 * R[mij])));
        });
      } else {
        static_for<(KL == 2 ? 4 : 1)>([&](auto hh) {
          constexpr int m = decltype(hh)::value;
          V[m] = pf_fma(b.A[i], R[m], b.h * R[herm_add(m, i)]);
        });
      }
      if constexpr (KL == 2) {
        T U[3], W[3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const T hv = kh * V[1 + x];
          U[x] = mkb * pf_fma(k.B[x], V[0], hv);
          W[x] = k.fa * pf_fma(k.A[x], V[0], hv);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const T G = gam(i, j, c, d);
            dY[c] = pf_fma(G, U[d], dY[c]);
            dY[d] = pf_fma(G, W[c], dY[d]);
          }
      } else {
        const T u = mkb * V[0];
#pragma unroll
        for (int c = 0; c < 3; ++c) dY[c] = pf_fma(gam(i, j, c, 0), u, dY[c]);
      }
    });
  const T mka = mone * k.fa;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    g[x] += pf_fma(b.fa, dP[x], dX[x]);
    g[3 + x] += pf_fma(b.fb, dP[x], mone * dX[x]);
    g[6 + x] += pf_fma(mka, dP[x], dY[x]);
  }
}

// FP operations of md_gradient (an FMA counts as two), from the loops above.
constexpr int md_flops(int bl, int kl) {
  const bool bb = bl == 2;
  const int L = bl + kl, nb = bb ? 3 : 1, ncd = kl == 2 ? 9 : (kl == 1 ? 3 : 1);
  int n = ncd * ((bb ? 54 : 8 * bl) + (bb ? 10 : 4) * 4 * kl);  // Hermite densities
  for (int m = 1; m <= L + 1; ++m) n += 2 * (herm_count(m) - 1);
  n += 8 * herm_count(L);
  if (bl > 0) n += ncd * ((bb ? 4 : 1) * (kl == 2 ? 7 : 3 * kl) + (bb ? 57 : 7));
  if (kl > 0) n += 3 * nb * ((kl == 2 ? 4 : 1) * (bb ? 7 : 3) + (bb ? 4 : 0) + (kl == 2 ? 57 : 7));
  return n + 56;
}

}  // namespace pyfacc

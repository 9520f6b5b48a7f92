// Dense per-molecule work of the batched engine.  One thread block per
// molecule; every n x n product is computed by the block itself on the FP64
// tensor cores (mma.sync m8n8k4) from L1/L2-resident operands (the
// matrices of a molecule of up to 160 basis functions are at most 200 KB),
// the TC2 iterate stays in shared memory, reductions go through shared
// memory, and nothing returns to the host between the Fock build and the
// next build density.
//
// The SCF step follows the single-molecule engine (rscf.f90:118-156 with
// DIIS and purification): F = H + J - K/2, E = 1/2 sum P (H + F), the DIIS
// error X (F P S - S P F) X, Pulay extrapolation over up to 8 stored
// matrices, F' = X F X, TC2 purification of F' to the projector on the nocc
// lowest orbitals, P = 2 X P' X.  X = S^{-1/2} (Loewdin orthogonalisation,
// from a coupled Newton-Schulz iteration, so no eigensolver is needed).
#include <cuda_runtime.h>

#include <climits>
#include <cmath>

#include "batch.h"

namespace pyfacc {

namespace {

__device__ __forceinline__ double red_op(double a, double b, bool mx) { return mx ? fmax(a, b) : a + b; }

// Block-wide sum (mx = false) or maximum; every thread receives the result.
__device__ double blk_reduce(double v, bool mx) {
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = red_op(v, __shfl_xor_sync(0xffffffffu, v, o), mx);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = red[l < nw ? l : 0];
  if (l >= nw && !mx) r = 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = red_op(r, __shfl_xor_sync(0xffffffffu, r, o), mx);
  __syncthreads();
  return r;
}

__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// The t-th 16 x 16 tile of the upper triangle of nm x nm tiles.
__device__ __forceinline__ void upper_tile(int t, int nm, int& ti, int& tj) {
  ti = 0;
  while (t >= nm - ti) t -= nm - ti++;
  tj = ti + t;
}

// C = alpha A B for n x n matrices with rows lda, ldb, ldc apart, on the FP64
// tensor cores: a warp owns 16 x 16 output tiles, four m8n8k4 products per
// two fragments of A and two of B.  The kernel is bound by the fragments'
// loads (L1 tag lookups: a fragment of four rows of 64 bytes takes four, one
// of eight rows of 32 bytes eight) where the 8 x 8 tiles it had before paid
// two fragments per product: 3.9 -> 0.80 ms a step for 256 molecules of 28 to
// 112 functions together with the purification below, 2.5 -> 0.54 ms for 64.  Hence AT: A is given
// transposed (a symmetric A is its own transpose; TS stores a result that is
// the next product's A).  SYM = 1 or -1: the result is symmetric or
// antisymmetric, only its upper triangle is computed.  A, B, C may be global
// or shared; C must not alias A or B.  Ends with a block barrier.
//
// Fragments of m8n8k4 (f64, row.col): lane l holds A[l/4][l%4],
// B[l%4][l/4] and C[l/4][2(l%4)], C[l/4][2(l%4)+1].
template <bool AT, int SYM, bool TS>
__device__ void bgemm(int n, const double* A, int lda, const double* B, int ldb, double* C, int ldc, double alpha) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nm = (n + 15) >> 4, ntile = SYM ? nm * (nm + 1) / 2 : nm * nm;
  for (int tile = warp; tile < ntile; tile += nwarp) {
    int ti = tile / nm, tj = tile - ti * nm;
    if (SYM) upper_tile(tile, nm, ti, tj);
    const int i0 = ti << 4, j0 = tj << 4;
    // rows of A and columns of B beyond n repeat the last one; their results
    // are not stored
    const int ia0 = min(i0 + g, n - 1), ia1 = min(i0 + 8 + g, n - 1);
    const int jb0 = min(j0 + g, n - 1), jb1 = min(j0 + 8 + g, n - 1);
    const double* pa0 = A + (AT ? (size_t)t * lda + ia0 : (size_t)ia0 * lda + t);
    const double* pa1 = A + (AT ? (size_t)t * lda + ia1 : (size_t)ia1 * lda + t);
    const double* pb0 = B + (size_t)t * ldb + jb0;
    const double* pb1 = B + (size_t)t * ldb + jb1;
    const int sa = AT ? 4 * lda : 4, sb = 4 * ldb;
    double acc[2][2][2] = {};
    auto step = [&](double a0, double a1, double b0, double b1) {
      mma_f64(acc[0][0][0], acc[0][0][1], a0, b0);
      mma_f64(acc[0][1][0], acc[0][1][1], a0, b1);
      mma_f64(acc[1][0][0], acc[1][0][1], a1, b0);
      mma_f64(acc[1][1][0], acc[1][1][1], a1, b1);
    };
    int k = 0;
#pragma unroll 4
    for (; k + 4 <= n; k += 4) {
      step(*pa0, *pa1, *pb0, *pb1);
      pa0 += sa; pa1 += sa; pb0 += sb; pb1 += sb;
    }
    if (k < n) {  // the last one to three k
      const bool in = k + t < n;
      step(in ? *pa0 : 0.0, in ? *pa1 : 0.0, in ? *pb0 : 0.0, in ? *pb1 : 0.0);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = i0 + 8 * r + g, col = j0 + 8 * c + 2 * t + h;
          if (row >= n || col >= n || (SYM && row > col)) continue;
          const double v = SYM < 0 && row == col ? 0.0 : alpha * acc[r][c][h];
          C[TS ? (size_t)col * ldc + row : (size_t)row * ldc + col] = v;
          if (SYM && row != col) C[(size_t)col * ldc + row] = SYM > 0 ? v : -v;
        }
  }
  __syncthreads();
}

// Rows of the shared-memory matrix: whole 16 x 16 tiles, 4 bank pairs apart
// (the eight rows of a fragment, four words each, then meet no bank twice).
__host__ __device__ constexpr int xs_rows(int n) { return (n + 15) & ~15; }
__host__ __device__ constexpr int xs_ld(int n) { return xs_rows(n) + 4; }

// TC2 purification (Niklasson 2002) of the orthogonalised Fock matrix Fp:
// xs (shared memory, rows xs_ld(n) apart) <- projector onto the nocc lowest
// eigenvectors.  The iterate stays in xs, zero-padded to whole tiles; X^2 of
// the upper triangle's tiles is accumulated in registers, up to TC2_TILES per
// warp, and xs is updated in place behind a barrier, with both triangles
// stored (X^T = X: the fragments of B are rows as well) and Tr X and Tr X^2
// (the square sum) taken along.  The step choice and the stopping rule are
// those of the single-molecule kernels (Tr X - Tr X^2 < 1e-9 at the right
// trace, then two more steps).  Returns the steps taken, or -1 without
// convergence.
constexpr int TC2_TILES = 4;  // 55 tiles at n = 160 (BATCH_NBF_MAX) on 16 warps
__device__ int tc2(int n, int nocc, const double* Fp, double* xs) {
  __shared__ double red[2][32];
  const int np = xs_rows(n), ld = xs_ld(n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (nocc <= 0 || nocc >= n) {
    for (int i = warp; i < n; i += nw)
      for (int j = lane; j < n; j += 32) xs[i * ld + j] = (nocc > 0 && i == j) ? 1.0 : 0.0;
    __syncthreads();
    return 0;
  }
  double lo = 1e300, hi = -1e300;
  for (int i = warp; i < n; i += nw) {
    double r = 0.0;
    for (int j = lane; j < n; j += 32)
      if (j != i) r += fabs(Fp[(size_t)i * n + j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    const double d = Fp[(size_t)i * n + i];
    lo = fmin(lo, d - r);
    hi = fmax(hi, d + r);
  }
  lo = -blk_reduce(-lo, true);
  hi = blk_reduce(hi, true);
  const double sc = 1.0 / fmax(hi - lo, 1e-300);
  double t1 = 0.0, t2 = 0.0;
  for (int i = warp; i < np; i += nw)
    for (int j = lane; j < np; j += 32) {
      double v = 0.0;
      if (i < n && j < n) v = ((i == j ? hi : 0.0) - Fp[(size_t)i * n + j]) * sc;
      if (i == j) t1 += v;
      t2 += v * v;
      xs[i * ld + j] = v;
    }
  t1 = blk_reduce(t1, false);
  t2 = blk_reduce(t2, false);
  const int g = lane >> 2, t = lane & 3;
  const int nm = np >> 4, ntile = nm * (nm + 1) / 2;
  int tij[TC2_TILES], mine = 0;
#pragma unroll
  for (int u = 0; u < TC2_TILES; ++u) {
    int ti = 0, tj = 0;
    if (warp + u * nw < ntile) {
      upper_tile(warp + u * nw, nm, ti, tj);
      mine = u + 1;
    }
    tij[u] = ti << 20 | tj << 4;
  }
  int countdown = 0;
  for (int k = 0; k < 200; ++k) {
    double acc[TC2_TILES][2][2][2];
#pragma unroll
    for (int u = 0; u < TC2_TILES; ++u) {
      if (u >= mine) break;
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[u][q >> 2][(q >> 1) & 1][q & 1] = 0.0;
      const double* pa = xs + ((tij[u] >> 16) + g) * ld + t;
      const double* pb = xs + ((tij[u] & 0xffff) + g) * ld + t;
#pragma unroll 2
      for (int kk = 0; kk < n; kk += 4) {
        const double a0 = pa[kk], a1 = pa[kk + 8 * ld], b0 = pb[kk], b1 = pb[kk + 8 * ld];
        mma_f64(acc[u][0][0][0], acc[u][0][0][1], a0, b0);
        mma_f64(acc[u][0][1][0], acc[u][0][1][1], a0, b1);
        mma_f64(acc[u][1][0][0], acc[u][1][0][1], a1, b0);
        mma_f64(acc[u][1][1][0], acc[u][1][1][1], a1, b1);
      }
    }
    bool finish = false;
    if (countdown > 0) {
      if (--countdown == 0) finish = true;
    } else if (t1 - t2 < 1e-9 && fabs(t1 - nocc) < 1e-6) {
      countdown = 2;
    }
    // X <- X^2 takes the trace to t2, X <- 2X - X^2 to 2 t1 - t2
    double a = 2.0, b = -1.0;
    if (fabs(t2 - nocc) < fabs(2.0 * t1 - t2 - nocc)) { a = 0.0; b = 1.0; }
    __syncthreads();  // every product has been read
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int u = 0; u < TC2_TILES; ++u) {
      if (u >= mine) break;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int row = (tij[u] >> 16) + 8 * (q >> 2) + g, col = (tij[u] & 0xffff) + 8 * ((q >> 1) & 1) + 2 * t + (q & 1);
        if (row > col) continue;
        const double v = a * xs[row * ld + col] + b * acc[u][q >> 2][(q >> 1) & 1][q & 1];
        xs[row * ld + col] = v;
        xs[col * ld + row] = v;
        if (row == col) s1 += v;
        s2 += row == col ? v * v : 2.0 * v * v;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      red[0][warp] = s1;
      red[1][warp] = s2;
    }
    __syncthreads();
    if (finish) return k + 1;
    t1 = lane < nw ? red[0][lane] : 0.0;
    t2 = lane < nw ? red[1][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    }
  }
  return -1;
}

// Pulay DIIS solve: B c = 0 with sum c = 1 over the m <= 8 slots in use,
// Gaussian elimination with partial pivoting on the bordered system.  One
// warp, lane r holds row r and the right-hand side; returns c_r in lane r and
// whether the system was solvable.
__device__ bool diis_solve(int m, const double* B, int ldb, const int* use, double& c) {
  constexpr int Q = BATCH_DIIS_MAX + 1;
  const unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31, q = m + 1;
  double scl = lane < m ? fabs(B[use[lane] * ldb + use[lane]]) : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) scl = fmax(scl, __shfl_xor_sync(ALL, scl, o));
  scl = scl > 0.0 ? 1.0 / scl : 1.0;
  double A[Q], b = lane == m ? -1.0 : 0.0;
#pragma unroll
  for (int j = 0; j < Q; ++j) {
    A[j] = 0.0;
    if (lane < m && j < m) A[j] = B[use[lane] * ldb + use[j]] * scl;
    else if (lane < q && j < q && lane != j) A[j] = -1.0;
  }
  bool ok = true;
#pragma unroll
  for (int col = 0; col < Q; ++col) {
    if (col >= q) break;
    // the largest of column col at or below the diagonal, the first of equals
    double v = lane >= col && lane < q ? fabs(A[col]) : -1.0;
    int piv = lane;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(ALL, v, o);
      const int op = __shfl_xor_sync(ALL, piv, o);
      if (ov > v || (ov == v && op < piv)) {
        v = ov;
        piv = op;
      }
    }
    piv = __shfl_sync(ALL, piv, 0);
    const int from = lane == col ? piv : (lane == piv ? col : lane);
    double f = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      A[k] = __shfl_sync(ALL, A[k], from);
      if (k < col) continue;
      const double p = __shfl_sync(ALL, A[k], col);
      if (k == col) {
        ok = ok && !(fabs(p) < 1e-300);
        f = lane > col ? A[k] / p : 0.0;
      }
      A[k] -= f * p;
    }
    b = __shfl_sync(ALL, b, from);
    b -= f * __shfl_sync(ALL, b, col);
  }
  c = 0.0;
#pragma unroll
  for (int r = Q - 1; r >= 0; --r) {
    if (r >= q) continue;
    const double x = __shfl_sync(ALL, b / A[r], r);
    if (lane == r) c = x;
    if (lane < r) b -= A[r] * x;
  }
  return __all_sync(ALL, ok && (lane >= m || isfinite(c)));
}

struct MolPtrs {
  int n, n2;
  const double *S, *H, *X;
  double *F, *J, *K, *Jd, *Kd, *P, *Db, *T1, *T2, *T3;
};

__device__ __forceinline__ MolPtrs mol_ptrs(const BatchDenseArgs& a, const BatchMolDev& d) {
  MolPtrs p;
  p.n = d.nbf;
  p.n2 = d.nbf * d.nbf;
  const size_t o = (size_t)d.mat_off;
  p.S = a.S + o; p.H = a.H + o; p.X = a.X + o;
  p.F = a.F + o; p.J = a.J + o; p.K = a.K + o; p.Jd = a.Jd + o; p.Kd = a.Kd + o;
  p.P = a.P + o; p.Db = a.Db + o; p.T1 = a.T1 + o; p.T2 = a.T2 + o; p.T3 = a.T3 + o;
  return p;
}

// P = 2 X P' X of the TC2 projector of F' = X Fsrc X; T1 and T3 are
// overwritten, the result goes to out.  Returns the TC2 steps or -1.
__device__ int density_from_fock(const MolPtrs& p, int nocc, const double* Fsrc, double* xs, double* out) {
  const int n = p.n;
  bgemm<true, 0, true>(n, p.X, n, Fsrc, n, p.T3, n, 1.0);  // (X F)^T
  bgemm<true, 1, false>(n, p.T3, n, p.X, n, p.T1, n, 1.0);
  const int steps = tc2(n, nocc, p.T1, xs);
  if (steps < 0) return -1;
  bgemm<true, 0, true>(n, p.X, n, xs, xs_ld(n), p.T3, n, 1.0);  // (X P')^T
  bgemm<true, 1, false>(n, p.T3, n, p.X, n, out, n, 2.0);
  return steps;
}

}  // namespace

// ---------------------------------------------------------------------------
// X = S^{-1/2}: coupled Newton-Schulz iteration Y0 = S/c, Z0 = I,
// T = (3I - Z Y)/2, Y <- Y T, Z <- T Z, which converges to Y = (S/c)^{1/2},
// Z = (S/c)^{-1/2} when the spectrum of S/c lies in (0, 1] (c = the largest
// absolute row sum of S, a bound on its largest eigenvalue).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(BATCH_THREADS) batch_lowdin_kernel(const BatchDenseArgs a, double* Xout) {
  const int m = blockIdx.x;
  const BatchMolDev d = a.mol[m];
  const MolPtrs p = mol_ptrs(a, d);
  const int n = p.n, n2 = p.n2;
  double c = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double r = 0.0;
    for (int j = 0; j < n; ++j) r += fabs(p.S[(size_t)i * n + j]);
    c = fmax(c, r);
  }
  c = blk_reduce(c, true);
  double* Y = p.T1;
  double* Z = p.T2;
  double* Tm = p.T3;
  double* fr = p.F;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int i = idx / n, j = idx - (idx / n) * n;
    Y[idx] = p.S[idx] / c;
    Z[idx] = (i == j) ? 1.0 : 0.0;
  }
  __syncthreads();
  bool ok = false;
  for (int it = 0; it < 100; ++it) {
    bgemm<false, 0, false>(n, Z, n, Y, n, Tm, n, 1.0);
    double dev = 0.0;
    for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
      const int i = idx / n, j = idx - (idx / n) * n;
      const double v = Tm[idx], e = (i == j) ? 1.0 : 0.0;
      dev = fmax(dev, fabs(v - e));
      Tm[idx] = 1.5 * e - 0.5 * v;
    }
    dev = blk_reduce(dev, true);
    bgemm<false, 0, false>(n, Y, n, Tm, n, fr, n, 1.0);
    { double* t = Y; Y = fr; fr = t; }
    bgemm<false, 0, false>(n, Tm, n, Z, n, fr, n, 1.0);
    { double* t = Z; Z = fr; fr = t; }
    if (dev < 1e-13) {
      ok = true;
      break;
    }
  }
  const double rs = 1.0 / sqrt(c);
  double* Xm = Xout + (size_t)d.mat_off;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int i = idx / n, j = idx - (idx / n) * n;
    Xm[idx] = 0.5 * (Z[idx] + Z[(size_t)j * n + i]) * rs;
  }
  if (threadIdx.x == 0 && !ok) a.st[m].failed = 1;
}

__global__ void batch_guess_kernel(const BatchDenseArgs a, const double* __restrict__ occ) {
  const int m = blockIdx.x;
  const BatchMolDev d = a.mol[m];
  double* P = a.P + (size_t)d.mat_off;
  const int n = d.nbf;
  for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
    const int i = idx / n, j = idx - (idx / n) * n;
    P[idx] = (i == j) ? occ[d.occ_off + i] : 0.0;
  }
}

// Start of the SCF: per-molecule state, zero J/K accumulators, the starting
// density (core guess: purification of F = H; otherwise P already holds the
// atomic-occupation guess) and Db = P for the first (full) build.
__global__ void __launch_bounds__(BATCH_THREADS) batch_init_kernel(const BatchDenseArgs a, int core_guess) {
  extern __shared__ double xs_sh[];
  const int m = blockIdx.x;
  const BatchMolDev d = a.mol[m];
  BatchMolState& st = a.st[m];
  const MolPtrs p = mol_ptrs(a, d);
  const int failed = st.failed;
  __syncthreads();
  if (threadIdx.x == 0) {
    st.E = st.E_prev = st.err = st.dD = st.E_final = 0.0;
    for (int k = 0; k < BATCH_DIIS_MAX * BATCH_DIIS_MAX; ++k) st.B[k] = 0.0;
    for (int k = 0; k < BATCH_DIIS_MAX; ++k) st.age[k] = -1;
    st.iter = st.head = st.converged = st.tc2_steps = 0;
    st.done = failed;
  }
  for (int idx = threadIdx.x; idx < p.n2; idx += blockDim.x) {
    p.J[idx] = 0.0;
    p.K[idx] = 0.0;
    p.Jd[idx] = 0.0;
    p.Kd[idx] = 0.0;
  }
  __syncthreads();
  if (!failed && core_guess) {
    const int steps = density_from_fock(p, d.nocc, p.H, xs_sh, p.P);
    if (steps < 0 && threadIdx.x == 0) {
      st.failed = 1;
      st.done = 1;
    }
    __syncthreads();
  }
  const bool skip = failed || st.done;
  for (int idx = threadIdx.x; idx < p.n2; idx += blockDim.x) p.Db[idx] = skip ? 0.0 : p.P[idx];
}

// One SCF step after the J/K build of Db (partial J, K in Jd, Kd).
__global__ void __launch_bounds__(BATCH_THREADS) batch_step_kernel(const BatchDenseArgs a) {
  extern __shared__ double xs_sh[];
  __shared__ double bro[BATCH_DIIS_MAX], coef[BATCH_DIIS_MAX];
  __shared__ int nuse, use_slot[BATCH_DIIS_MAX];
  const int m = blockIdx.x;
  BatchMolState& st = a.st[m];
  if (st.done || st.failed) return;
  const BatchMolDev d = a.mol[m];
  const MolPtrs p = mol_ptrs(a, d);
  const int n = p.n, n2 = p.n2;
  const int it = st.iter + 1;
  const double E_prev = st.E_prev, dD_prev = st.dD;
  const bool built_full = a.built_full != 0;
  const int ld = xs_ld(n), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // ---- J, K (J = Jh + Jh^T of the build), F and the energy of P; the halves
  // are transposed through shared memory
  double e = 0.0;
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j < n; j += 32) xs_sh[i * ld + j] = p.Jd[(size_t)i * n + j];
  __syncthreads();
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j < n; j += 32) {
      const size_t q = (size_t)i * n + j;
      p.J[q] = (built_full ? 0.0 : p.J[q]) + xs_sh[i * ld + j] + xs_sh[j * ld + i];
      p.Jd[q] = 0.0;
    }
  __syncthreads();
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j < n; j += 32) xs_sh[i * ld + j] = p.Kd[(size_t)i * n + j];
  __syncthreads();
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j < n; j += 32) {
      const size_t q = (size_t)i * n + j;
      const double kn = (built_full ? 0.0 : p.K[q]) + xs_sh[i * ld + j] + xs_sh[j * ld + i];
      p.K[q] = kn;
      p.Kd[q] = 0.0;
      const double h = p.H[q], f = h + p.J[q] - 0.5 * kn;
      p.F[q] = f;
      e += p.P[q] * (h + f);
    }
  const double E = 0.5 * blk_reduce(e, false);
  // ---- DIIS error X (F P S - S P F) X  (S P F = (F P S)^T)
  bgemm<true, 0, true>(n, p.F, n, p.P, n, p.T3, n, 1.0);  // (F P)^T
  bgemm<true, 0, false>(n, p.T3, n, p.S, n, xs_sh, ld, 1.0);
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j <= i; j += 32) {
      const double v = xs_sh[i * ld + j] - xs_sh[j * ld + i];
      xs_sh[i * ld + j] = v;
      xs_sh[j * ld + i] = -v;
    }
  __syncthreads();
  bgemm<true, 0, true>(n, p.X, n, xs_sh, ld, p.T3, n, 1.0);
  bgemm<true, -1, false>(n, p.T3, n, p.X, n, p.T1, n, 1.0);
  double em = 0.0;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) em = fmax(em, fabs(p.T1[idx]));
  em = blk_reduce(em, true);
  const double dE = fabs(E - E_prev);
  if (threadIdx.x == 0 && a.max_err) atomicMax(a.max_err, (unsigned long long)__double_as_longlong(em));
  bool conv = !a.coarse && dE < a.e_tol && em < a.eps_diis;
  if (a.eps_density > 0) conv = conv && it > 1 && dD_prev < a.eps_density;
  if (threadIdx.x == 0) {
    st.E = E;
    st.err = em;
    st.iter = it;
    st.E_final = E;
  }
  if (conv || it >= a.max_iter) {
    if (threadIdx.x == 0) {
      st.done = 1;
      st.converged = conv ? 1 : 0;
    }
    for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) p.Db[idx] = 0.0;
    return;
  }
  // ---- DIIS: store F and the error, overlaps, extrapolate
  const double* Fuse = p.F;
  if (a.ndiis > 0) {
    double* dF = a.diis + d.diis_off;
    double* dEr = dF + (size_t)a.ndiis * n2;
    const int slot = st.head;
    // the stored F and error, and the error's products with all stored ones
    // (a slot in use, or this one) in one pass
    bool used[BATCH_DIIS_MAX];
    double v[BATCH_DIIS_MAX];
#pragma unroll
    for (int k = 0; k < BATCH_DIIS_MAX; ++k) {
      used[k] = k < a.ndiis && k != slot && st.age[k] >= 0;
      v[k] = 0.0;
    }
    for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
      const double x = p.T1[idx];
      dF[(size_t)slot * n2 + idx] = p.F[idx];
      dEr[(size_t)slot * n2 + idx] = x;
#pragma unroll
      for (int k = 0; k < BATCH_DIIS_MAX; ++k)
        if (used[k]) v[k] += x * dEr[(size_t)k * n2 + idx];
        else if (k == slot) v[k] += x * x;
    }
#pragma unroll
    for (int k = 0; k < BATCH_DIIS_MAX; ++k)
      if (used[k] || k == slot) {
        const double w = blk_reduce(v[k], false);
        if (threadIdx.x == 0) bro[k] = w;
      }
    __syncthreads();  // every thread has read the slot ages before warp 0 changes them
    if (warp == 0) {
      const int D = BATCH_DIIS_MAX;
      if (lane == 0) {
        st.age[slot] = it;
        for (int k = 0; k < a.ndiis; ++k)
          if (st.age[k] >= 0) {
            st.B[slot * D + k] = bro[k];
            st.B[k * D + slot] = bro[k];
          }
        st.head = (slot + 1) % a.ndiis;
        nuse = 0;
      }
      if (lane < BATCH_DIIS_MAX) coef[lane] = 0.0;
      __syncwarp();
      int age = lane < a.ndiis ? st.age[lane] : -1;
      // drop the oldest vectors until the system is solvable
      while (true) {
        const unsigned in_use = __ballot_sync(0xffffffffu, age >= 0);
        const int nu = __popc(in_use);
        if (nu < 2) break;
        if (age >= 0) use_slot[__popc(in_use & ((1u << lane) - 1u))] = lane;
        __syncwarp();
        double c;
        const bool solved = diis_solve(nu, st.B, D, use_slot, c);
        if (solved) {
          if (lane < nu) coef[use_slot[lane]] = c;
          if (lane == 0) nuse = nu;
          break;
        }
        // the ages differ: iterations
        int oldest = age >= 0 ? age : INT_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) oldest = min(oldest, __shfl_xor_sync(0xffffffffu, oldest, o));
        if (age == oldest) {
          age = -1;
          st.age[lane] = -1;
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (nuse >= 2) {
      for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
        double v = 0.0;
        for (int k = 0; k < a.ndiis; ++k)
          if (coef[k] != 0.0) v += coef[k] * dF[(size_t)k * n2 + idx];
        p.T2[idx] = v;
      }
      __syncthreads();
      Fuse = p.T2;
    }
  }
  // ---- new density: Fuse (F or T2) is read before T2 is reused
  double* Pn = p.T2;
  const int steps = density_from_fock(p, d.nocc, Fuse, xs_sh, Pn);
  if (steps < 0) {
    if (threadIdx.x == 0) {
      st.failed = 1;
      st.done = 1;
    }
    for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) p.Db[idx] = 0.0;
    return;
  }
  // ---- next build density: P_new - P for an incremental build, else P_new
  // (a full rebuild of an incremental run sets Db = P before its build)
  const bool next_full = !a.incremental;
  double dd = 0.0;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const double pn = Pn[idx], diff = pn - p.P[idx];
    dd += diff * diff;
    p.Db[idx] = next_full ? pn : diff;
    p.P[idx] = pn;
  }
  dd = blk_reduce(dd, false);
  if (threadIdx.x == 0) {
    st.dD = sqrt(dd);
    st.E_prev = E;
    st.tc2_steps += steps;
    atomicAdd(a.active, 1);
  }
}

// F and E of the converged density after a full build of Db = P (the FP64
// polish of mixed precision); J, K, F are replaced, E -> st.E_final.
__global__ void __launch_bounds__(BATCH_THREADS) batch_polish_kernel(const BatchDenseArgs a) {
  const int m = blockIdx.x;
  BatchMolState& st = a.st[m];
  if (st.failed || !st.done) return;
  const BatchMolDev d = a.mol[m];
  const MolPtrs p = mol_ptrs(a, d);
  const int n = p.n, n2 = p.n2;
  double e = 0.0;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int i = idx / n, j = idx - (idx / n) * n;
    const size_t t = (size_t)j * n + i;
    const double jn = p.Jd[idx] + p.Jd[t], kn = p.Kd[idx] + p.Kd[t];
    p.J[idx] = jn;
    p.K[idx] = kn;
    const double f = p.H[idx] + jn - 0.5 * kn;
    p.F[idx] = f;
    e += p.P[idx] * (p.H[idx] + f);
  }
  e = blk_reduce(e, false);
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    p.Jd[idx] = 0.0;
    p.Kd[idx] = 0.0;
  }
  if (threadIdx.x == 0) st.E_final = 0.5 * e;
}

// Db = P for the molecules that finished (FP64 polish build), 0 otherwise.
__global__ void batch_polish_density_kernel(const BatchDenseArgs a) {
  const int m = blockIdx.x;
  const BatchMolState& st = a.st[m];
  const BatchMolDev d = a.mol[m];
  const MolPtrs p = mol_ptrs(a, d);
  const bool use = st.done && !st.failed;
  for (int idx = threadIdx.x; idx < p.n2; idx += blockDim.x) p.Db[idx] = use ? p.P[idx] : 0.0;
}

// W = 1/2 P F P (RHF energy-weighted density at convergence).
__global__ void __launch_bounds__(BATCH_THREADS) batch_wdens_kernel(const BatchDenseArgs a, double* out) {
  const int m = blockIdx.x;
  const BatchMolDev d = a.mol[m];
  const MolPtrs p = mol_ptrs(a, d);
  bgemm<true, 0, false>(p.n, p.F, p.n, p.P, p.n, p.T1, p.n, 1.0);
  bgemm<true, 0, false>(p.n, p.P, p.n, p.T1, p.n, out + (size_t)d.mat_off, p.n, 0.5);
}

__global__ void batch_dmax_kernel(int ns_max, const int4* __restrict__ mt, const int* __restrict__ bf_off,
                                  const int* __restrict__ nfun, const double* __restrict__ D, float* __restrict__ dm) {
  const int m = blockIdx.y;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ns_max * ns_max) return;
  const int4 t = mt[m];  // {first shell, ns, mat_off, nbf}
  const int a = idx / ns_max, b = idx - (idx / ns_max) * ns_max;
  float* out = dm + (size_t)m * ns_max * ns_max;
  if (a >= t.y || b >= t.y) {
    out[idx] = 0.0f;
    return;
  }
  const int sa = t.x + a, sb = t.x + b;
  double mx = 0.0;
  for (int i = 0; i < nfun[sa]; ++i)
    for (int j = 0; j < nfun[sb]; ++j)
      mx = fmax(mx, fabs(D[(size_t)t.z + (size_t)(bf_off[sa] + i) * t.w + bf_off[sb] + j]));
  out[idx] = (float)mx;
}

static constexpr size_t xs_bytes(int nmax) { return (size_t)xs_rows(nmax) * xs_ld(nmax) * sizeof(double); }

void batch_set_smem() {
  allow_smem(batch_init_kernel, xs_bytes(BATCH_NBF_MAX));
  allow_smem(batch_step_kernel, xs_bytes(BATCH_NBF_MAX));
}

__global__ void __launch_bounds__(BATCH_THREADS) batch_full_density_kernel(const BatchDenseArgs a) {
  const int m = blockIdx.x;
  const BatchMolState& st = a.st[m];
  if (st.done || st.failed) return;
  const BatchMolDev d = a.mol[m];
  const size_t n2 = (size_t)d.nbf * d.nbf;
  const double* P = a.P + d.mat_off;
  double* Db = a.Db + d.mat_off;
  for (size_t idx = threadIdx.x; idx < n2; idx += blockDim.x) Db[idx] = P[idx];
}

void launch_batch_full_density(int nmol, const BatchDenseArgs& a, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_full_density_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_lowdin(int nmol, const BatchDenseArgs& a, double* Xout, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_lowdin_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a, Xout);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_guess(int nmol, const BatchDenseArgs& a, const double* occ, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_guess_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a, occ);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_init(int nmol, const BatchDenseArgs& a, int core_guess, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_init_kernel<<<nmol, BATCH_THREADS, xs_bytes(a.smem_nmax), s>>>(a, core_guess);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

// ---------------------------------------------------------------------------
// Control of the whole-SCF graph (one thread each).
// ---------------------------------------------------------------------------
__global__ void batch_ctl_select_kernel(const BatchScfCtl* __restrict__ c, int* __restrict__ report,
                                        cudaGraphConditionalHandle variant) {
  report[0] = 0;  // active molecules
  report[1] = 0;
  report[2] = 0;  // largest DIIS error (bits of a double, two ints)
  report[3] = 0;
  cudaGraphSetConditional(variant, (unsigned)c->variant);
}

__global__ void batch_ctl_update_kernel(BatchScfCtl* __restrict__ c, const int* __restrict__ report,
                                        cudaGraphConditionalHandle loop) {
  c->counts[c->variant] += 1;
  const int it = ++c->it;
  const int active = report[0];
  const double err = __longlong_as_double(*reinterpret_cast<const long long*>(report + 2));
  bool go = active > 0;
  if (go && c->coarse && (err < c->coarse_err || it >= c->coarse_max_iter)) {
    c->coarse = 0;
    c->restart = 1;
  }
  if (it >= c->max_iter) go = false;
  if (go) {
    int v;
    if (c->coarse) {
      v = G_CINC;
    } else {
      const bool full = !c->incremental || c->restart || c->since_full + 1 >= c->rebuild_every;
      c->since_full = full ? 0 : c->since_full + 1;
      c->restart = 0;
      v = full ? G_FULL : G_INC;
    }
    c->variant = v;
  }
  c->stop = go ? 0 : 1;
  cudaGraphSetConditional(loop, go ? 1u : 0u);
}

void add_batch_select_node(cudaGraph_t g, cudaGraphNode_t* node, BatchScfCtl* ctl, int* report,
                           cudaGraphConditionalHandle variant) {
  const BatchScfCtl* c = ctl;
  void* args[] = {&c, &report, &variant};
  cudaKernelNodeParams p{};
  p.func = reinterpret_cast<void*>(batch_ctl_select_kernel);
  p.gridDim = dim3(1);
  p.blockDim = dim3(1);
  p.kernelParams = args;
  PF_CUDA(cudaGraphAddKernelNode(node, g, nullptr, 0, &p));
}

void add_batch_update_node(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* dep, BatchScfCtl* ctl,
                           const int* report, cudaGraphConditionalHandle loop) {
  void* args[] = {&ctl, &report, &loop};
  cudaKernelNodeParams p{};
  p.func = reinterpret_cast<void*>(batch_ctl_update_kernel);
  p.gridDim = dim3(1);
  p.blockDim = dim3(1);
  p.kernelParams = args;
  PF_CUDA(cudaGraphAddKernelNode(node, g, dep, 1, &p));
}

void launch_batch_step(int nmol, const BatchDenseArgs& a, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_step_kernel<<<nmol, BATCH_THREADS, xs_bytes(a.smem_nmax), s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_polish(int nmol, const BatchDenseArgs& a, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_polish_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_polish_density(int nmol, const BatchDenseArgs& a, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_polish_density_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_wdens(int nmol, const BatchDenseArgs& a, double* out, cudaStream_t s) {
  if (nmol <= 0) return;
  batch_wdens_kernel<<<nmol, BATCH_THREADS, 0, s>>>(a, out);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_dmax(int nmol, int ns_max, const int4* mt, const int* bf_off, const int* nfun, const double* D,
                       float* dm, cudaStream_t s) {
  if (nmol <= 0 || ns_max <= 0) return;
  dim3 grid((ns_max * ns_max + 127) / 128, nmol), block(128);
  batch_dmax_kernel<<<grid, block, 0, s>>>(ns_max, mt, bf_off, nfun, D, dm);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace pyfacc

// Pair and task lists of the batched engine, built on the device.
//
// Pairs of a class are sorted by molecule, then by Schwarz factor Q
// (descending), so the kets a bra reaches are a prefix of its molecule's
// segment of the ket class: Q_bra Q_ket >= thresh, and in mixed precision
// the FP64 part the prefix with Q_bra Q_ket >= fp32_thresh (for the
// gradient, >= grad_fp32_thresh); for equal classes only kets up to the bra
// itself are canonical.  One thread per bra
// finds the prefixes by binary search (batch_ranges_kernel); one block per
// (class combination, precision, task width) turns the ket ranges into task
// offsets with a block-wide exclusive scan (batch_scan_kernel) and reports
// the task and quartet counts, which the host reads once.
#include <cuda_runtime.h>

#include "batch.h"

namespace pyfacc {

namespace {

__device__ __forceinline__ int q_prefix(const double4* __restrict__ geom, int base, int n, double qb, double t) {
  if (t <= 0) return n;
  int lo = 0, hi = n;  // count of j with qb * Q_j >= t, Q descending
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (qb * geom[base + mid].w >= t) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(256) batch_ranges_kernel(const BatchRangeArgs A) {
  const BatchRangeList& L = A.l[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.nb) return;
  const int bp = L.bra_base + i;
  const double qb = A.geom[bp].w;
  const int m = A.info2[bp].z;  // molecule of the bra
  const int ks = L.seg_k[m], nk = L.seg_k[m + 1] - ks;
  int mm = q_prefix(A.geom, L.ket_base + ks, nk, qb, A.thresh);
  if (L.same) mm = min(mm, i - L.seg_b[m] + 1);
  const int m64 = min(q_prefix(A.geom, L.ket_base + ks, nk, qb, A.fp32_thresh), mm);
  const int mg = min(q_prefix(A.geom, L.ket_base + ks, nk, qb, A.grad_fp32_thresh), mm);
  L.lo[3][i] = ks;
  L.hi[3][i] = ks + mg;
  L.lo[4][i] = ks + mg;
  L.hi[4][i] = ks + mm;
  L.lo[0][i] = ks;
  L.hi[0][i] = ks + mm;
  L.lo[1][i] = ks;
  L.hi[1][i] = ks + m64;
  L.lo[2][i] = ks + m64;
  L.hi[2][i] = ks + mm;
}

__global__ void __launch_bounds__(1024) batch_scan_kernel(const BatchScanArgs A) {
  const BatchScanList& L = A.l[blockIdx.x];
  __shared__ int wsum[32];
  __shared__ long long wq[32];
  __shared__ int carry;
  __shared__ long long qcarry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) {
    carry = 0;
    qcarry = 0;
  }
  __syncthreads();
  for (int base = 0; base < L.nb; base += blockDim.x) {
    const int i = base + threadIdx.x;
    int cnt = 0;
    long long nq = 0;
    if (i < L.nb) {
      const int len = L.hi[i] - L.lo[i];
      cnt = (len + L.width - 1) / L.width;
      nq = len;
    }
    int v = cnt;
    long long vq = nq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
      vq += __shfl_xor_sync(0xffffffffu, vq, o);
    }
    if (lane == 31) wsum[w] = v;
    if (lane == 0) wq[w] = vq;
    __syncthreads();
    if (w == 0) {
      int x = lane < nw ? wsum[lane] : 0;
      long long xq = lane < nw ? wq[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
        xq += __shfl_xor_sync(0xffffffffu, xq, o);
      }
      wsum[lane] = x;  // inclusive over warps
      if (lane == 0) wq[0] = xq;
    }
    __syncthreads();
    const int excl = carry + (w > 0 ? wsum[w - 1] : 0) + v - cnt;
    if (i < L.nb) L.toff[i] = excl;
    const int total = wsum[nw - 1];
    const long long tq = wq[0];
    __syncthreads();
    if (threadIdx.x == 0) {
      carry += total;
      qcarry += tq;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    L.toff[L.nb] = carry;
    A.ntasks[blockIdx.x] = carry;
    A.nquartets[blockIdx.x] = qcarry;
  }
}

// The pair lists of all molecules, a block per molecule: with the numbers of s
// and p shells before every shell, and the sums of their primitive counts, the
// place of a pair within its class and its first primitive pair are products
// and triangle numbers.  256 water clusters: 10 MB of lists written here instead
// of on the host and copied, setup 18.4 -> 13.6 ms.
__global__ void __launch_bounds__(256) batch_pairs_kernel(const BatchPairArgs A) {
  extern __shared__ int sh[];
  const int m = blockIdx.x;
  const int4 mt = A.mt[m];  // {first shell, ns, mat_off, nbf}
  const int ns = mt.y;
  // per shell: type, primitives, then of each type before it: shells,
  // primitives, squares of the primitives
  int *l = sh, *n = l + A.ns_max, *cnt = n + A.ns_max, *sum = cnt + 2 * A.ns_max, *sq = sum + 2 * A.ns_max;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    l[i] = A.desc[mt.x + i].x > 0 ? 1 : 0;
    n[i] = A.nprim[mt.x + i];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    int c = 0, s = 0, q = 0;
    for (int i = 0; i < ns; ++i) {
      cnt[2 * i + threadIdx.x] = c;
      sum[2 * i + threadIdx.x] = s;
      sq[2 * i + threadIdx.x] = q;
      if (l[i] == (int)threadIdx.x) {
        ++c;
        s += n[i];
        q += n[i] * n[i];
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ns * (ns + 1) / 2; t += blockDim.x) {
    int i = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while (i * (i + 1) / 2 > t) --i;
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    const int j = t - i * (i + 1) / 2, li = l[i], lj = l[j], c = li + lj;
    int k = cnt[2 * j + lj], z = n[i] * sum[2 * j + lj];  // within row i
    if (c == 1) {
      k += cnt[2 * i] * cnt[2 * i + 1];
      z += sum[2 * i] * sum[2 * i + 1];
    } else {
      k += cnt[2 * i + li] * (cnt[2 * i + li] + 1) / 2;
      // (twice the result may pass 2^31)
      const unsigned s = sum[2 * i + li];
      z += (int)((s * s + (unsigned)sq[2 * i + li]) / 2);
    }
    k += A.pair_off[c * A.nmol + m];
    z += A.prim_off[c * A.nmol + m];
    const int a = li < lj ? j : i, b = li < lj ? i : j;
    A.pl0[k] = make_int4(mt.x + a, mt.x + b, z, mt.x);
    A.pl1[k] = make_int4(mt.z, mt.w, m, m * A.ns_max * A.ns_max);
  }
}

}  // namespace

void launch_batch_pairs(const BatchPairArgs& a, cudaStream_t s) {
  if (a.nmol <= 0) return;
  batch_pairs_kernel<<<a.nmol, 256, 8 * (size_t)a.ns_max * sizeof(int), s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_ranges(const BatchRangeArgs& a, int nlists, int nb_max, cudaStream_t s) {
  if (nlists <= 0 || nb_max <= 0) return;
  dim3 grid((nb_max + 255) / 256, nlists), block(256);
  batch_ranges_kernel<<<grid, block, 0, s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

void launch_batch_scans(const BatchScanArgs& a, int nlists, cudaStream_t s) {
  if (nlists <= 0) return;
  batch_scan_kernel<<<nlists, 1024, 0, s>>>(a);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace pyfacc

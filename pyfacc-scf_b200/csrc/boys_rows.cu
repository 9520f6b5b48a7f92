// The split kernels' Boys tables (boys_rows.cuh): interpolated on the host in
// long double, one copy per device.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "boys_rows.cuh"
#include "engine.h"
#include "split.cuh"

namespace pyfacc {

namespace {

__device__ BoysRows<double> g_br64[BR_LMAX + 1];
__device__ BoysRows<float> g_br32[BR_LMAX + 1];
constexpr int MAX_DEVICES = 64;
const char* g_addr[MAX_DEVICES][2] = {};  // of g_br64, g_br32

// F_m near and above T = 0 in long double (also for the small negative
// arguments of the first row's interpolation points).
long double boys_ld(int m, long double T) {
  long double sum = 0.0L;
  if (T < 1.0L) {
    long double t = 1.0L;
    for (int k = 0; k < 40; ++k) {
      sum += t / (2 * m + 2 * k + 1);
      t *= -T / (k + 1);
    }
    return sum;
  }
  long double t = 1.0L / (2 * m + 1);
  for (int k = 1; k < 2000 && t > sum * 1e-22L; ++k) {
    sum += t;
    t *= 2.0L * T / (2 * m + 2 * k + 1);
  }
  return expl(-T) * sum;
}

// Monomial coefficients in x of the polynomial that interpolates F_L(c + x)
// at the n Chebyshev points of |x| <= r.
void row_coefficients(int L, long double c, long double r, int n, long double* out) {
  std::vector<long double> f(n), a(n), t0(n, 0.0L), t1(n, 0.0L), t2(n);
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int i = 0; i < n; ++i) f[i] = boys_ld(L, c + r * cosl(pi * (i + 0.5L) / n));
  for (int j = 0; j < n; ++j) {
    a[j] = 0.0L;
    for (int i = 0; i < n; ++i) a[j] += f[i] * cosl(pi * j * (i + 0.5L) / n);
    a[j] *= (j == 0 ? 1.0L : 2.0L) / n;
  }
  for (int j = 0; j < n; ++j) out[j] = 0.0L;
  t0[0] = 1.0L;
  t1[1] = 1.0L;
  for (int j = 0; j < n; ++j) {  // t0 = T_j in powers of x / r
    for (int k = 0; k <= j; ++k) out[k] += a[j] * t0[k];
    for (int k = 0; k < n; ++k) t2[k] = (k > 0 ? 2.0L * t1[k - 1] : 0.0L) - t0[k];
    t0 = t1;
    t1 = t2;
  }
  long double s = 1.0L;
  for (int k = 0; k < n; ++k, s *= r) out[k] /= s;
}

// One function value per thread, for the tests: the table's F_0 .. F_L, the
// far limit's (far_setup at |PQ|^2 = T with rho = 1), or far_rsqrt and br_expm.
template <int L, bool FP32> __device__ void split_values(int what, double x, double* out) {
  if (what == 0) {
    if constexpr (FP32) {
      F2 F[L + 1];
      boys_rows<L>(g_br32[L], F2((float)x), F);
      for (int m = 0; m <= L; ++m) out[m] = F[m].v.x;
    } else {
      boys_rows<L>(g_br64[L], x, out);
    }
  } else if (what == 1) {
    using T = typename std::conditional<FP32, F2, double>::type;
    PrimGeo<T> g;
    const T PQ[3] = {T(typename Scalar<T>::R(sqrt(x))), T(0.0f), T(0.0f)};
    far_setup<T, L>(PQ, T(typename Scalar<T>::R(0.88622692545275801365)), T(0.5f), T(0.5f), g);
    for (int m = 0; m <= L; ++m) {
      if constexpr (FP32) out[m] = g.I[m].v.x;
      else out[m] = g.I[m];
    }
  } else if (what == 2) {
    if constexpr (FP32) out[0] = far_rsqrt((float)x);
    else out[0] = far_rsqrt(x);
  } else {
    out[0] = br_expm(x);
  }
}
template <bool FP32>
__global__ void split_values_kernel(int what, int L, int n, const double* __restrict__ x, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double* o = out + (size_t)i * (L + 1);
  switch (L) {
    case 0: split_values<0, FP32>(what, x[i], o); break;
    case 1: split_values<1, FP32>(what, x[i], o); break;
    case 2: split_values<2, FP32>(what, x[i], o); break;
    case 3: split_values<3, FP32>(what, x[i], o); break;
    default: split_values<4, FP32>(what, x[i], o); break;
  }
}

}  // namespace

void launch_split_values(int what, bool fp32, int L, int n, const double* x, double* out, cudaStream_t s) {
  if (n <= 0) return;
  if (fp32) split_values_kernel<true><<<(n + 127) / 128, 128, 0, s>>>(what, L, n, x, out);
  else split_values_kernel<false><<<(n + 127) / 128, 128, 0, s>>>(what, L, n, x, out);
  PF_CUDA(cudaGetLastError());
  count_launch();
}

// The tables of the current device (called once per device, under the lock of
// ensure_boys_tables).
void upload_boys_rows(int device) {
  static std::vector<BoysRows<double>> t64;
  static std::vector<BoysRows<float>> t32;
  if (t64.empty()) {
    t64.resize(BR_LMAX + 1);
    t32.resize(BR_LMAX + 1);
    for (int L = 0; L <= BR_LMAX; ++L)
      for (int r = 0; r < BR_ROWS; ++r) {
        long double c[BR_N64];
        const long double h = br_step<double>(L);
        row_coefficients(L, r * h, 0.5L * h, BR_N64, c);
        for (int j = 0; j < BR_N64; ++j) {
          const double v = (double)c[j];
          unsigned long long u;
          std::memcpy(&u, &v, 8);
          t64[L].hi[j][r] = (unsigned)(u >> 32);
          t64[L].lo[j][r] = (unsigned)u;
        }
        const long double hf = (float)br_step<float>(L);
        row_coefficients(L, r * hf, 0.5L * hf, BR_N32, c);
        for (int j = 0; j < BR_N32; ++j) t32[L].c[j][r] = (float)c[j];
      }
  }
  PF_CUDA(cudaMemcpyToSymbol(g_br64, t64.data(), sizeof(g_br64)));
  PF_CUDA(cudaMemcpyToSymbol(g_br32, t32.data(), sizeof(g_br32)));
  void *p64 = nullptr, *p32 = nullptr;
  PF_CUDA(cudaGetSymbolAddress(&p64, g_br64));
  PF_CUDA(cudaGetSymbolAddress(&p32, g_br32));
  if (device >= MAX_DEVICES) throw Error(PYFACC_ERR_INVALID, "device ordinal beyond " + std::to_string(MAX_DEVICES));
  g_addr[device][0] = static_cast<const char*>(p64);
  g_addr[device][1] = static_cast<const char*>(p32);
}

const void* boys_rows_table(bool fp32, int L) {
  int device = 0;
  PF_CUDA(cudaGetDevice(&device));
  return g_addr[device][fp32] + (size_t)L * (fp32 ? sizeof(BoysRows<float>) : sizeof(BoysRows<double>));
}

}  // namespace pyfacc

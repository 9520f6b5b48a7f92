// The split kernels' Boys tables (boys_rows.cuh): interpolated on the host in
// long double, one copy per device.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "boys_rows.cuh"
#include "engine.h"

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

}  // namespace

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

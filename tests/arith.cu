// The kernels' own arithmetic element by element, for test_gpu_arith.py (built
// by it with nvcc into a library of its own).
#include <cuda_runtime.h>

#include "../brams_gb300/csrc/lw_table.cuh"
#include "../brams_gb300/csrc/sw_kernel.cuh"

namespace {

template <class F>
__global__ void each(long long n, F f) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) f(i);
}
template <class F>
int run(long long n, F f) {
  each<<<1216, 256>>>(n, f);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? cudaDeviceSynchronize() : e;
}

}  // namespace

extern "C" {

// rtrnmc's quotient and table index of optical depths
int arith_tbl(const float* od, float* q, int* itr, long long n) {
  return run(n, [=] __device__(long long i) {
    q[i] = gb::tbl_quotient(od[i]);
    itr[i] = gb::tbl_index(od[i]);
  });
}

// div_mid against the operator: quotients 2^ea s(i) / 2^eb t over all 2^23 significands s for each of n significands t
// (of t's bits); bad[0] += the number that differ, bad[1] the last such divisor's bits
int arith_div_rows(const unsigned* t, int ea, int eb, unsigned* bad, long long n) {
  return run(n << 23, [=] __device__(long long i) {
    const float b = __uint_as_float((unsigned)(127 + eb) << 23 | (t[i >> 23] & 0x7fffffu));
    const float a = __uint_as_float((unsigned)(127 + ea) << 23 | (unsigned)(i & 0x7fffff));
    if (gbsw::div_mid(a, b) != a / b) atomicAdd(bad, 1u), bad[1] = __float_as_uint(b);
  });
}
// the same for all 2^23 divisors, each with the n dividends a; exact[d] = 1 where rcp_mid of the divisor rounds as 1 / b
int arith_div_cols(const float* a, int eb, unsigned* bad, unsigned char* exact, int n) {
  return run(1LL << 23, [=] __device__(long long i) {
    const float b = __uint_as_float((unsigned)(127 + eb) << 23 | (unsigned)i);
    exact[i] = gbsw::rcp_mid(b) == 1.0f / b;
    for (int k = 0; k < n; ++k)
      if (gbsw::div_mid(a[k], b) != a[k] / b) atomicAdd(bad, 1u), bad[1] = __float_as_uint(b);
  });
}
// and for pairs
int arith_div(const float* a, const float* b, float* q, float* ref, long long n) {
  return run(n, [=] __device__(long long i) { q[i] = gbsw::div_mid(a[i], b[i]), ref[i] = a[i] / b[i]; });
}

// fp64: reciprocal, square root, division by the constants of setcoef, and the operators
int arith_f64(const double* x, double* rcp, double* root, double* c15, double* c36, double* c72, long long n) {
  return run(n, [=] __device__(long long i) {
    const double v = x[i];
    rcp[2 * i] = gbsw::rcp64(v), rcp[2 * i + 1] = 1.0 / v;
    root[2 * i] = gbsw::sqrt64(v), root[2 * i + 1] = sqrt(v);
    c15[2 * i] = gbsw::div_c(v, 15.0), c15[2 * i + 1] = v / 15.0;
    c36[2 * i] = gbsw::div_c(v, 36.0), c36[2 * i + 1] = v / 36.0;
    c72[2 * i] = gbsw::div_c(v, 7.2), c72[2 * i + 1] = v / 7.2;
  });
}

// float -> double by bits, all 2^32 patterns (values that are not numbers aside): bad[0] of f2d_fast, bad[1] of
// f2d_scaled (finite values; its product with 2^896 is exact)
int arith_f2d(unsigned* bad) {
  return run(1LL << 32, [=] __device__(long long i) {
    const float x = __uint_as_float((unsigned)i);
    if (x != x) return;
    if (__double_as_longlong(gbsw::f2d_fast(x)) != __double_as_longlong((double)x)) atomicAdd(bad, 1u);
    if (isfinite(x) && __double_as_longlong(gbsw::f2d_scaled(x) * 0x1p896) != __double_as_longlong((double)x))
      atomicAdd(bad + 1, 1u);
  });
}

// the table directory of this library's copy: the exponential table alone, at the start of the blob
int arith_sw_table(double bpade) {
  gbsw::SwTab t{};
  t.exp_tbl = 0;
  t.bpade = bpade;
  t.bpadef = (float)bpade;
  return gbsw::sw_set_tab(t);
}
int arith_index64(const double* ze, int* itr, long long n) {
  return run(n, [=] __device__(long long i) { itr[i] = gbsw::tbl_index64(ze[i]); });
}
// reftra_f with the fast divisions and with the operators: out[side][i][pref, prefd, ptra, ptrad, dbt], for either sky
int arith_reftra(const float* T, const float* zg, const float* mu, const float* tau, const float* zw, const float* zco,
                 float* out, int total, long long n) {
  return run(n, [=] __device__(long long i) {
    float* f = out + 5 * i;
    float* s = out + 5 * (n + i);
    if (total) {
      gbsw::reftra_f<true, true>(T, zg[i], mu[i], tau[i], zw[i], zco[i], f[0], f[1], f[2], f[3], f[4]);
      gbsw::reftra_f<false, true>(T, zg[i], mu[i], tau[i], zw[i], zco[i], s[0], s[1], s[2], s[3], s[4]);
    } else {
      gbsw::reftra_f<true, false>(T, zg[i], mu[i], tau[i], zw[i], zco[i], f[0], f[1], f[2], f[3], f[4]);
      gbsw::reftra_f<false, false>(T, zg[i], mu[i], tau[i], zw[i], zco[i], s[0], s[1], s[2], s[3], s[4]);
    }
  });
}

}  // extern "C"

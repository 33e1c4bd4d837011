// The kernels' own arithmetic element by element, for test_gpu_arith.py (built
// by it with nvcc into a library of its own).
#include <cuda_runtime.h>

#include "../brams_gb300/csrc/lw_table.cuh"

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

}  // extern "C"

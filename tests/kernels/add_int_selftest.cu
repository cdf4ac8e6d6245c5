// Self-test of fdfx::add_int against the hardware addition.  Test infrastructure: built by the GPU tests,
// not part of the library.
#include <cuda_runtime.h>

#include "fdf_exact.cuh"

namespace {

__global__ void k_check(const double *__restrict__ a, const double *__restrict__ b, long long n,
                        unsigned long long *bad) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const double got = fdfx::add_int(a[t], b[t]), want = __dadd_rn(a[t], b[t]);
    if (fdfx::ubits(got) != fdfx::ubits(want) && !(fdfx::is_nan(got) && fdfx::is_nan(want))) atomicAdd(bad, 1ull);
  }
}

}  // namespace

// Counts the mismatches over n operand pairs (host arrays).  Returns a CUDA error code.
extern "C" int fdf_test_add_int(const double *a, const double *b, long long n, unsigned long long *bad) {
  double *d = nullptr;
  unsigned long long *c = nullptr;
  cudaError_t e = cudaMalloc((void **)&d, 16 * n);
  if (e == cudaSuccess) e = cudaMalloc((void **)&c, 8);
  if (e == cudaSuccess) e = cudaMemset(c, 0, 8);
  if (e == cudaSuccess) e = cudaMemcpy(d, a, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_check<<<256, 256>>>(d, d + n, n, c);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(bad, c, 8, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(c);
  return (int)e;
}

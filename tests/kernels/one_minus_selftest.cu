// Self-test of fdfx::one_minus against the hardware subtraction and of fdfx::mul_int against the
// hardware multiply at the operands their bit arithmetic turns on.  Test infrastructure: built by the
// GPU tests, not part of the library.
#include <cuda_runtime.h>

#include "fdf_exact.cuh"

namespace {

__device__ __forceinline__ bool same(double a, double b) {
  const unsigned long long ua = fdfx::ubits(a), ub = fdfx::ubits(b);
  return ua == ub || (fdfx::is_nan(a) && fdfx::is_nan(b));
}

__global__ void k_check(const double *__restrict__ a, const double *__restrict__ b, long long n,
                        unsigned long long *bad) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    if (!same(fdfx::one_minus(a[t]), __dsub_rn(1.0, a[t]))) atomicAdd(&bad[0], 1ull);
    if (!same(fdfx::mul_int(a[t], b[t]), __dmul_rn(a[t], b[t]))) atomicAdd(&bad[1], 1ull);
  }
}

}  // namespace

// Counts the mismatches over n operand pairs (host arrays).  Returns a CUDA error code.
extern "C" int fdf_test_one_minus(const double *a, const double *b, long long n, unsigned long long *bad) {
  double *d = nullptr;
  unsigned long long *c = nullptr;
  cudaError_t e = cudaMalloc((void **)&d, 16 * n);
  if (e == cudaSuccess) e = cudaMalloc((void **)&c, 16);
  if (e == cudaSuccess) e = cudaMemset(c, 0, 16);
  if (e == cudaSuccess) e = cudaMemcpy(d, a, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_check<<<256, 256>>>(d, d + n, n, c);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(bad, c, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(c);
  return (int)e;
}

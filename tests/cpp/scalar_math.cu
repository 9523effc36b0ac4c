// Evaluates the branch-free reciprocals, quotient and root of the kernels
// (csrc/physics.cuh) on arrays of host values.
#include <cuda_runtime.h>

#include "physics.cuh"

namespace {

__global__ void eval_kernel(int op, const double* a, const double* b, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = op == 0   ? dgsem::recip(a[i])
           : op == 1 ? dgsem::quotient(a[i], b[i])
           : op == 2 ? dgsem::root(a[i])
                     : dgsem::recip_ulp(a[i]);
}

}  // namespace

extern "C" int scalar_math_eval(int op, const double* a, const double* b, double* out, int n) {
  double* d = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  if (op < 0 || op > 3 || n < 1 || cudaMalloc(&d, 3 * bytes) != cudaSuccess) return 1;
  cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  eval_kernel<<<(n + 255) / 256, 256>>>(op, d, d + n, d + 2 * (size_t)n, n);
  cudaMemcpy(out, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaGetLastError();
  cudaFree(d);
  return e == cudaSuccess ? 0 : 1;
}

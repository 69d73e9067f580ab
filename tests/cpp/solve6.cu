// kf_solve6 for n systems, on the host (compiled as C++) or on the device (as CUDA).
#include <cstdint>
#include "kf_solve6.cuh"

#ifdef __CUDACC__
__global__ void solve_kernel(const double* c, const double* b, double* x, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) kf_solve6(c + 21 * k, b + 6 * k, x + 6 * k);
}

extern "C" int solve_all(const double* c, const double* b, double* x, int n) {
  double* d = nullptr;
  if (cudaMalloc((void**)&d, (size_t)n * 33 * 8) != cudaSuccess) return 1;
  cudaMemcpy(d, c, (size_t)n * 21 * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(d + (size_t)n * 21, b, (size_t)n * 6 * 8, cudaMemcpyHostToDevice);
  solve_kernel<<<(n + 127) / 128, 128>>>(d, d + (size_t)n * 21, d + (size_t)n * 27, n);
  const bool ok = cudaMemcpy(x, d + (size_t)n * 27, (size_t)n * 6 * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? 0 : 1;
}
#else
extern "C" int solve_all(const double* c, const double* b, double* x, int n) {
  for (int k = 0; k < n; ++k) kf_solve6(c + 21 * k, b + 6 * k, x + 6 * k);
  return 0;
}
#endif

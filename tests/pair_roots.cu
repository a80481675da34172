// The FP64 roots of the pair arithmetic beside CUDA's own, for
// test_pair_roots.py: out holds 7 columns of n values.
#include <cstdint>

#include "sph_device.cuh"

namespace {
__global__ void k_pair_roots(const double* a, const double* b, int64_t n, double* out) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  out[i] = sph::rsqrt_approx(a[i]);
  out[n + i] = sph::frsqrt<double>(a[i]);
  out[2 * n + i] = 1.0 / sqrt(a[i]);
  out[3 * n + i] = sph::fsqrt<double>(a[i]);
  out[4 * n + i] = sqrt(a[i]);
  out[5 * n + i] = sph::froot_ratio(a[i], b[i]);
  out[6 * n + i] = sqrt(a[i] / b[i]);
}
}  // namespace

// a, b: n host values each, out: 7 n host values
extern "C" int pair_roots(const double* a, const double* b, int64_t n, double* out) {
  double* d = nullptr;
  if (n < 1 || cudaMalloc(&d, sizeof(double) * 9 * n) != cudaSuccess) return 1;
  cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k_pair_roots<<<int((n + 255) / 256), 256>>>(d, d + n, n, d + 2 * n);
  const cudaError_t e = cudaMemcpy(out, d + 2 * n, sizeof(double) * 7 * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}

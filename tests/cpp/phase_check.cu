// The device functions of csrc/phase.cuh on arrays, for a test to compare with
// CUDA's own and with extended precision.
#include <cuda_runtime.h>

#include "phase.cuh"

namespace {

__global__ void roots_kernel(const double* x, double* y, double* ref, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = bemgpu::newton_sqrt(x[i], rsqrt(x[i]));
  ref[i] = sqrt(x[i]);
}

template <int NS, int NC>
__global__ void phases_kernel(const double* x, double* s, double* c, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bemgpu::sincos_taylor<NS, NC>(x[i], s[i], c[i]);
}

// out0 and out1 of n values from x, by run(device x, device out0, device out1)
template <typename F>
int on_device(const double* x, double* out0, double* out1, int n, F run) {
  const size_t bytes = (size_t)n * sizeof(double);
  double* d = nullptr;
  if (cudaMalloc((void**)&d, 3 * bytes) != cudaSuccess) return 1;
  cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice);
  run(d, d + n, d + 2 * (size_t)n);
  cudaMemcpy(out0, d + n, bytes, cudaMemcpyDeviceToHost);
  cudaMemcpy(out1, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() != cudaSuccess;
}

}  // namespace

extern "C" int phase_roots(const double* x, double* y, double* ref, int n) {
  return on_device(x, y, ref, n, [n](const double* a, double* b, double* c) {
    roots_kernel<<<(n + 255) / 256, 256>>>(a, b, c, n);
  });
}

// the series for |x| <= 0.35 (wide = 0) or <= 1
extern "C" int phase_sincos(const double* x, double* s, double* c, int n, int wide) {
  return on_device(x, s, c, n, [n, wide](const double* a, double* b, double* d) {
    if (wide) phases_kernel<8, 9><<<(n + 255) / 256, 256>>>(a, b, d, n);
    else phases_kernel<6, 6><<<(n + 255) / 256, 256>>>(a, b, d, n);
  });
}

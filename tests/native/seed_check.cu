// Test harness (not part of the library): the FP64 reciprocal, quotient and
// square root with FP32 seeds and the FP32 sums of device_math.cuh on host
// arrays.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_math.cuh"

namespace {

__global__ void k_check(int64_t n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ r,
                        double* __restrict__ q, double* __restrict__ s, double* __restrict__ by) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = mgcfd::rcp_fast(b[i]);
  q[i] = mgcfd::div_fast(a[i], b[i]);
  s[i] = mgcfd::sqrt_fast(b[i]);
  by[i] = mgcfd::div_by(a[i], b[i], mgcfd::rcp_fast(b[i]));
}

// One row of m terms per thread.
__global__ void k_sum(int64_t n, int m, const float* __restrict__ x, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  mgcfd::Sum32 s = {};
  for (int j = 0; j < m; j++) mgcfd::sum32_add(s, x[i * m + j]);
  out[i] = mgcfd::sum32_value(s);
}

}  // namespace

extern "C" int sum_check(int64_t n, int m, const float* x, double* out) {
  float* d = nullptr;
  double* o = nullptr;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d), sizeof(float) * (size_t)(n * m));
  if (!e) e = cudaMalloc(reinterpret_cast<void**>(&o), sizeof(double) * (size_t)n);
  if (!e && !(e = cudaMemcpy(d, x, sizeof(float) * (size_t)(n * m), cudaMemcpyHostToDevice))) {
    k_sum<<<(unsigned)((n + 127) / 128), 128>>>(n, m, d, o);
    if (!(e = cudaGetLastError())) e = cudaMemcpy(out, o, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  cudaFree(o);
  return (int)e;
}

// Host buffers in (a, b) and out (1/b, a/b, sqrt(b), a/b by div_by); returns a cudaError_t value.
extern "C" int seed_check(int64_t n, const double* a, const double* b, double* r, double* q, double* s, double* by) {
  const size_t bytes = sizeof(double) * (size_t)n;
  double* d = nullptr;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d), 6 * bytes);
  if (e) return (int)e;
  if (!(e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice)) &&
      !(e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice))) {
    k_check<<<(unsigned)((n + 127) / 128), 128>>>(n, d, d + n, d + 2 * n, d + 3 * n, d + 4 * n, d + 5 * n);
    if (!(e = cudaGetLastError()) && !(e = cudaMemcpy(r, d + 2 * n, bytes, cudaMemcpyDeviceToHost)) &&
        !(e = cudaMemcpy(q, d + 3 * n, bytes, cudaMemcpyDeviceToHost)) &&
        !(e = cudaMemcpy(s, d + 4 * n, bytes, cudaMemcpyDeviceToHost)))
      e = cudaMemcpy(by, d + 5 * n, bytes, cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  return (int)e;
}

// The device functions of zq_recip.cuh over an array (tests/test_recip_gpu.py): the value
// and its relative error as the residual 1 - d y or (1 - q y^2) / 2 in exact products.
#include "zq_recip.cuh"

namespace {
__global__ void k_recip(const double* x, double* y, double* err, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = zq::recip(x[i]);
  err[i] = fma(-x[i], y[i], 1.0);
}
__global__ void k_recip_sqrt(const double* x, double* y, double* err, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = zq::recip_sqrt(x[i]);
  const double p = v * v, pl = fma(v, v, -p);
  y[i] = v;
  err[i] = 0.5 * (fma(-x[i], p, 1.0) - x[i] * pl);
}
}  // namespace

extern "C" int test_recip(int which, const double* x, double* y, double* err, long long n) {
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (which) k_recip_sqrt<<<blocks, 256>>>(x, y, err, n);
  else k_recip<<<blocks, 256>>>(x, y, err, n);
  const cudaError_t launch = cudaGetLastError();
  const cudaError_t done = cudaDeviceSynchronize();
  return launch != cudaSuccess ? (int)launch : (int)done;
}

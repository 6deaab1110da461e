// The scalar functions of the FP64 sweeps (gcs_physics.cuh), evaluated on the
// device for tests/test_sweep_math_gpu.py.
#include "gcs_physics.cuh"

namespace {

__global__ void k_eval(int which, long long n, const double *x, double *y, double *z) {
  using N = gcs::Num<double>;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  z[i] = 0.0;
  switch (which) {
    case 0: y[i] = N::rcp(x[i]); break;
    case 1: y[i] = N::rsqrt_(x[i]); break;
    case 2: y[i] = N::sqrt0(x[i]); break;
    default: N::erfc_exp(x[i], &y[i], &z[i]); break;
  }
}

}  // namespace

// which: 0 rcp, 1 rsqrt_, 2 sqrt0, 3 erfc_exp; host arrays of n values.
extern "C" int sweep_math(int which, long long n, const double *x, double *y, double *z) {
  double *d = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  if (n < 1 || cudaMalloc(&d, 3 * bytes) != cudaSuccess) return -1;
  bool ok = cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) k_eval<<<(unsigned)((n + 255) / 256), 256>>>(which, n, d, d + n, d + 2 * n);
  ok = ok && cudaGetLastError() == cudaSuccess &&
       cudaMemcpy(y, d + n, bytes, cudaMemcpyDeviceToHost) == cudaSuccess &&
       cudaMemcpy(z, d + 2 * n, bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? 0 : -1;
}

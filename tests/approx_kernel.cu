// rcp_f, rsqrt_f and sqrt_f on arrays, for test_gpu_approx.py.
#include "physics.cuh"

__global__ void k_approx(long n, const double* x, double* rcp, double* rsq, double* sq) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  rcp[t] = grb::rcp_f(x[t]);
  rsq[t] = grb::rsqrt_f(x[t]);
  sq[t] = grb::sqrt_f(x[t]);
}
extern "C" int approx(long n, const double* x, double* rcp, double* rsq, double* sq, void* stream) {
  k_approx<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, x, rcp, rsq, sq);
  return (int)cudaGetLastError();
}

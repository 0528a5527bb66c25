// The device arithmetic of pfgpu_device.cuh beside CUDA's division, for the
// tests: op 0 the reciprocal of b, 1 the quotient a / b, 2 the same in FP32.
#include <cuda_runtime.h>

#include "pfgpu_device.cuh"

using namespace pfgpu;

__global__ void k_check(int op, const double *a, const double *b, double *got, double *want,
                        long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (op == 0) {
      got[i] = fast_rcp(b[i]);
      want[i] = 1.0 / b[i];
    } else if (op == 1) {
      got[i] = rcp_far(b[i]) ? a[i] / b[i] : quotient_near(a[i], b[i]);
      want[i] = a[i] / b[i];
    } else {
      const float x = (float)a[i], y = (float)b[i];
      got[i] = rcp_far(y) ? x / y : quotient_near(x, y);
      want[i] = x / y;
    }
  }
}

// 1 where the operand takes the division
__global__ void k_far(int fp32, const double *b, double *far, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) far[i] = fp32 ? rcp_far((float)b[i]) : rcp_far(b[i]);
}

extern "C" int arith_check(int op, const double *a, const double *b, double *got, double *want,
                           long long n) {
  k_check<<<1184, 256>>>(op, a, b, got, want, n);
  return (int)cudaDeviceSynchronize();
}
extern "C" int arith_far(int fp32, const double *b, double *far, long long n) {
  k_far<<<(unsigned)((n + 255) / 256), 256>>>(fp32, b, far, n);
  return (int)cudaDeviceSynchronize();
}

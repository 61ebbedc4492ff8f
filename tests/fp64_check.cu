// Device harness for tests/test_gpu_fp64_roots.py: the step's reciprocal and
// square root beside CUDA's correctly rounded ones.
#include <cuda_runtime.h>

#include "hb_fp64.cuh"

__global__ void fp64_check_kernel(int n, const double *x, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = hb::rcp64(x[i]);
  out[n + i] = __drcp_rn(x[i]);
  out[2 * n + i] = hb::sqrt64(x[i]);
  out[3 * n + i] = __dsqrt_rn(x[i]);
}

// x[n] and out[4 n] on the device; returns the CUDA error code.
extern "C" int fp64_check(int n, const double *x, double *out, void *stream) {
  fp64_check_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(n, x, out);
  return (int)cudaGetLastError();
}

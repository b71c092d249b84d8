// Device build of the FP64 1/sqrt (fp64_math.cuh) beside CUDA's.
#include <cuda_runtime.h>

#include "fp64_math.cuh"

__global__ void k_rsqrt(int n, const double* x, double* own, double* cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  own[i] = ibem::rsqrt_h3(x[i]);
  cuda[i] = rsqrt(x[i]);
}

extern "C" int dr_rsqrt(int n, const double* x, double* own, double* cuda) {
  k_rsqrt<<<(n + 255) / 256, 256>>>(n, x, own, cuda);
  return (int)cudaDeviceSynchronize();
}

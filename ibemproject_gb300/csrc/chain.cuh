// Launches that overlap the end of the kernel before (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

#include "ibem_internal.h"

namespace ibem {

// Kernels that depend on each other and take a few microseconds each, as long as a launch (Arnoldi
// steps of small batches, the leaves of the FP32 LU): they are launched so that the successor's
// launch overlaps the end of its predecessor, and begin with chain_wait(): nothing is read or
// written before the predecessor has finished and its writes are visible.  A kernel of few CTAs
// (kChainCtas, two for each of GB300's 152 SMs) lets its successor's CTAs be set up as soon as its
// own have all started; one of many leaves that to their end, because CTAs set up early crowd
// onto the SMs that are free first.
// Solve of 64 particles 1.89 -> 1.52 ms, 12 quadratic realisations 15.8 -> 15.5 (17.2 with every
// successor set up early); mixed-precision LU of N = 16,800 (4,650 launches) 95.6 -> 88.0 ms.
constexpr unsigned kChainCtas = 304;
__device__ __forceinline__ void chain_wait() {
#ifdef __CUDA_ARCH__
  if (gridDim.x * gridDim.y * gridDim.z <= kChainCtas) cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
#endif
}
template <class... P, class... A>
inline void launch_chained_smem(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  count_launch();
  (void)cudaLaunchKernelEx(&c, k, P(a)...);   // its error is the thread's last error
}
template <class... P, class... A>
inline void launch_chained(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t st, A... a) {
  launch_chained_smem(k, grid, block, 0, st, a...);
}

}  // namespace ibem

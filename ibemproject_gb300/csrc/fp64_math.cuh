// FP64 1/sqrt for the kernels bound by the FP64 pipe (2 results per clock and SM on GB300).
#pragma once
#include <math.h>

#include "gen_sphere_common.cuh"

namespace ibem {

// The hardware's estimate (about 20 bits) and one step of Householder's third-order iteration:
// with e = 1 - x y^2, y (1 + e / 2 + 3 e^2 / 8) leaves a relative error of 5 e^3 / 16, below
// 2^-58.  The rounding of x y enters by half and that of the result in full: 1.54 2^-53 at
// most; measured over every exponent 1.14 2^-53 (CUDA's rsqrt 1.00).  Five FP64 operations.
// x = 0, infinite or subnormal gives NaN or infinity: callers evaluate a kernel that is
// singular there.
IBEM_HD IBEM_INLINE double rsqrt_h3(double x) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
#else
  return 1.0 / sqrt(x);
#endif
}

}  // namespace ibem

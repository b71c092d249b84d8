// Search key of the FP64 panels' pivots (solver.cu).
#pragma once
#include "gen_sphere_common.cuh"

namespace ibem {

// Key of a live entry in row q (< 2^IB), its upper word hi: greater for the greater |a|, and at equal
// size for the smaller row, so that one unsigned maximum picks the pivot; never 0.  The size has
// 14 bits of the mantissa, as in the FP32 panels, and what is left of 32 bits for the exponent:
// all of it for 128 rows, 2^-896, 2^-384 and 2^-128 to 2^127 for 256, 512 and 1,024 rows (of the
// equilibrated matrix); smaller and greater entries count as the range's ends.  In integers:
// a conversion to FP32 would be one more operation on the FP64 pipe.
template <int IB>
IBEM_HD IBEM_INLINE unsigned pivot_key64(unsigned hi, int q) {
  constexpr int E = 18 - IB;   // bits of the exponent
  constexpr unsigned lo = (E == 11 ? 0u : 1151u - (1u << E)) << 20, up = lo + (((1u << E) - 1u) << 20);
  unsigned h = hi & 0x7fffffffu;
  h = h < lo ? lo : h;
  h = h > up ? up : h;
  return ((((h - lo) >> 6) + 1u) << IB) | ((1u << IB) - 1u - (unsigned)q);
}

}  // namespace ibem

// Host build of the FP64 panels' pivot search key (pivot_key.cuh).
#include "pivot_key.cuh"

extern "C" unsigned hp_key64(int index_bits, unsigned hi, int q) {
  switch (index_bits) {
    case 7: return ibem::pivot_key64<7>(hi, q);
    case 8: return ibem::pivot_key64<8>(hi, q);
    case 9: return ibem::pivot_key64<9>(hi, q);
    default: return ibem::pivot_key64<10>(hi, q);
  }
}

// oic_occurrences.h -- positions in a hash block's occurrence array, as the seed kernel
// computes them; compiles for the host too, where the tests run it.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define OIC_OCC_FN __device__ __forceinline__
#else
#define OIC_OCC_FN inline
#endif

namespace oic {

// The first position of the run [start, end) whose block string is `from` or a later one
// (end: none).  A run ascends by string.  A block holds up to 2^32 - 1 occurrences, so the
// sum of two positions does not fit 32 bits.  strAt(p): the string of occurrence p.
template <class StrAt>
OIC_OCC_FN uint32_t first_occurrence_from(uint32_t start, uint32_t end, uint32_t from, StrAt strAt) {
  while (start < end) {
    const uint32_t mid = start + ((end - start) >> 1);
    if (strAt(mid) >= from) end = mid;
    else start = mid + 1;
  }
  return start;
}

}  // namespace oic

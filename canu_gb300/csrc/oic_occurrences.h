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

// Most match nodes of a ref strand in any seed configuration (node 0 stands for none).
constexpr uint32_t kSeedNodeCapMax = 1u << 22;

// The seeds of one ref offset: the occurrences of its k-mer's run [start, end) in string
// `from` or later ones; kTooManySeeds when there are nodeCap (<= kSeedNodeCapMax) or more.
// Such a strand cannot be held: the seeds of one offset lie on different diagonals or in
// different partners, so each of them ends in a match node of its own.  The kernel gives up
// the strand there and then; below that, the seeds of up to 1,024 offsets add up in 32 bits.
constexpr uint32_t kTooManySeeds = 0xffffffffu;
template <class StrAt>
OIC_OCC_FN uint32_t offset_seeds(uint32_t start, uint32_t end, uint32_t from, uint32_t nodeCap, StrAt strAt) {
  const uint32_t n = end - first_occurrence_from(start, end, from, strAt);
  return n < nodeCap ? n : kTooManySeeds;
}

}  // namespace oic

// Positions in the occurrence array, for tests/test_occurrences.py: the seed kernel's search
// on a synthetic array in which occurrence p lies in string p / div.
#include <cinttypes>
#include <cstdio>

#include "oic_occurrences.h"

int main() {
  uint32_t start, end, from, div;
  while (scanf("%" SCNu32 " %" SCNu32 " %" SCNu32 " %" SCNu32, &start, &end, &from, &div) == 4) {
    uint32_t outside = 0;
    const uint32_t p = oic::first_occurrence_from(start, end, from, [&](uint32_t i) {
      outside += i < start || i >= end;
      return i / div;
    });
    printf("%" PRIu32 " %" PRIu32 "\n", p, outside);
  }
}

// Positions in the occurrence array, for tests/test_occurrences.py: the seed kernel's search
// on a synthetic array in which occurrence p lies in string p / div ("s" lines), and its sum
// of the seeds of 256 ref offsets that all have the same run ("o" lines).
#include <cinttypes>
#include <cstdio>

#include "oic_occurrences.h"

int main() {
  char     what;
  uint32_t start, end, from, div;
  while (scanf(" %c %" SCNu32 " %" SCNu32 " %" SCNu32 " %" SCNu32, &what, &start, &end, &from, &div) == 5) {
    if (what == 'o') {
      uint32_t sum = 0, flagged = 0;
      for (int i = 0; i < 256; i++) {
        const uint32_t n = oic::offset_seeds(start, end, from, oic::kSeedNodeCapMax, [&](uint32_t p) { return p / div; });
        if (n == oic::kTooManySeeds) flagged++;
        else sum += n;
      }
      printf("%" PRIu32 " %" PRIu32 "\n", sum, flagged);
      continue;
    }
    uint32_t outside = 0;
    const uint32_t p = oic::first_occurrence_from(start, end, from, [&](uint32_t i) {
      outside += i < start || i >= end;
      return i / div;
    });
    printf("%" PRIu32 " %" PRIu32 "\n", p, outside);
  }
}

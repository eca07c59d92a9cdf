// The record pass's memory layout as text, for tests/test_store_layout.py.
#include <cstdio>

#include "oic_store_layout.h"

int main() {
  unsigned long long n, scr;
  unsigned maxID;
  while (scanf("%llu %u %llu", &n, &maxID, &scr) == 3) {
    const oic::StoreLayout l = oic::store_layout(n, maxID, scr);
    printf("%zu %zu %zu %zu %zu %zu %zu %zu %zu %zu %zu %zu %zu %zu %zu\n", l.in, l.keys, l.keep, l.pos, l.rec, l.k2,
           l.k3, l.idx, l.idx2, l.scr, l.cnt, l.a, l.aOff, l.out, l.bytes);
  }
}

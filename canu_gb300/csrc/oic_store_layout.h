// oic_store_layout.h -- the device memory of the overlap-store record pass: one allocation,
// the byte offset of each of its arrays.  Host code only.
#pragma once

#include <cstddef>
#include <cstdint>

namespace oic {

struct StoreLayout {
  size_t in, keys, keep, pos;      // dead once the kept copies are compacted: `out` lies over them
  size_t rec, k2, k3, idx, idx2, scr, cnt, a, aOff;
  size_t out;                      // the sorted records, as many as are kept (at most 2 n)
  size_t bytes;
};

// n input records, read IDs up to maxID, scr bytes of scan and sort scratch.
inline StoreLayout store_layout(uint64_t n, uint32_t maxID, size_t scr) {
  const size_t n2 = 2 * (size_t)n, ids = ((size_t)maxID + 2) * 4;
  size_t used = 0;
  const auto take = [&](size_t bytes) {
    const size_t at = used;
    used += (bytes + 255) & ~(size_t)255;
    return at;
  };
  StoreLayout l;
  l.in   = take((size_t)n * 24);
  l.keys = take(n2 * 8);
  l.keep = take((n2 + 1) * 4);
  l.pos  = take((n2 + 1) * 4);
  l.out  = l.in;                   // 48 n of the 56 n bytes so far
  l.rec  = take(n2 * 24);
  l.k2   = take(n2 * 8);
  l.k3   = take(n2 * 8);
  l.idx  = take(n2 * 4);
  l.idx2 = take(n2 * 4);
  l.scr  = take(scr);
  l.cnt  = take(8 * 8 + 4 * 4);    // 8 counters, then the compaction total
  l.a    = take(ids);
  l.aOff = take(ids);
  l.bytes = used;
  return l;
}

}  // namespace oic

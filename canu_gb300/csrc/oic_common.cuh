// oic_common.cuh -- shared device-side definitions of the GB300 overlapInCore engine.
//
// Read layout in HBM: every read is packed 2 bits per base (A=0 C=1 G=2 T=3, base i
// of a read at bits 2*(i%32) of 64-bit word i/32, the same order overlapInCore builds
// its k-mer keys in, Build_Hash_Index.C:347-350) in two strand arrays -- forward and
// reverse complement -- plus a parallel mask array with 0b11 at every N.  The DP reads the
// same bases as bit planes (word i: the low bits of bases 32i .. 32i+31, then their high
// bits, base 32i topmost), in which a comparison of 32 bases is four funnel shifts and two
// logic instructions, and the first difference a count of leading zeros.  Reads start on a
// word boundary and are separated by one zero guard word, so a 32-base window that runs off
// either end of a read stays inside the arrays.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace oic {

typedef unsigned long long u64;
typedef long long          i64;
typedef unsigned int       u32;

constexpr u32 kMaxReadLenBits = 21;                              // AS_MAX_READLEN_BITS
constexpr u32 kMaxReadLen     = (1u << kMaxReadLenBits) - 1;     // AS_MAX_READLEN
constexpr int kHopelessMatch  = 90;                              // overlapInCore.H:78
constexpr int kMaxDistinct    = 3;                               // overlapInCore.H:107
constexpr int kMinIntersect   = 10;                              // overlapInCore.H:120
constexpr int kShiftSlack     = 1;                               // overlapInCore.H:146
constexpr int kEntriesPerBucket = 21;                            // overlapInCore.H:58
constexpr u64 kEmptyKey       = ~0ull;

// Device error flags (bitwise OR into ctx->dErr).  Kernels never trap: they record
// the condition, skip the access and return.
enum : u32 {
  kErrBadBase      = 1u << 0,
  kErrArenaFull    = 1u << 1,   // DP traceback arena of a warp exhausted
  kErrBandWide     = 1u << 2,   // DP band wider than the shared-memory row buffer
  kErrRowsFull     = 1u << 3,   // more DP rows than the row-header capacity
  kErrNodePool     = 1u << 4,   // seed replay: node pool of a warp exhausted
  kErrPairTable    = 1u << 5,   // seed replay: pair table of a warp exhausted
  kErrOutNodes     = 1u << 6,   // global node output full
  kErrOutPairs     = 1u << 7,   // global pair output full
  kErrDeltaFull    = 1u << 8,
  kErrTableFull    = 1u << 9,   // k-mer table probe ran through every slot
  kErrInternal     = 1u << 10,
  kErrNodesPerPair = 1u << 11
};

// Packed reads (device pointers).
struct ReadsDev {
  const u64 *fwd;       // forward strand words
  const u64 *rc;        // reverse-complement strand words
  const u64 *nfwd;      // N masks (0b11 per N) for the forward strand
  const u64 *nrc;
  const uint2 *pfwd;    // bit planes of the forward strand (x low bits, y high bits)
  const uint2 *prc;
  const u64 *wordOff;   // first word of read i (0-based index = ID-1)
  const u32 *len;
  const u32 *lib;
  const unsigned char *hasN;
  u32 nReads;
};

// One read strand viewed as a base sequence: base i is base i of the read's first word.
struct SeqView {
  const uint2 *p;  // the read's first bit-plane word in its strand array
  const u64 *nm;   // its first N-mask word; nullptr when the read has no N
};

// A read strand and its reverse complement.
struct ReadView {
  SeqView f, c;
};

__device__ __forceinline__ ReadView make_view(const ReadsDev &R, u32 readIdx, int rev) {
  ReadView v;
  const u64  wo = R.wordOff[readIdx];
  const bool hn = R.hasN[readIdx] != 0;
  const SeqView a = {R.pfwd + wo, hn ? R.nfwd + wo : nullptr}, b = {R.prc + wo, hn ? R.nrc + wo : nullptr};
  v.f = rev ? b : a;
  v.c = rev ? a : b;
  return v;
}

// 32 bases starting at global base index g (base g in bits 0-1).  Both words are
// always read (the arrays end with two spare words), and the high word's shift is
// split in two so that sh = 0 needs no branch: (hi << 1) << 63 is 0.
__device__ __forceinline__ u64 load_win(const u64 *w, i64 g) {
  const i64 wi = g >> 5;
  const int sh = (int)(g & 31) * 2;
  const u64 lo = __ldg(w + wi);
  const u64 hi = __ldg(w + wi + 1);
  return (lo >> sh) | ((hi << 1) << (63 - sh));
}

// The same for base g of one read (w = the read's first word; -32 < g: the guard word
// before every read keeps g - 31 in bounds), in 32-bit index arithmetic.
__device__ __forceinline__ u64 load_win32(const u64 *w, int g) {
  const int wi = g >> 5;
  const int sh = (g & 31) * 2;
  const u64 lo = __ldg(w + wi);
  const u64 hi = __ldg(w + wi + 1);
  return (lo >> sh) | ((hi << 1) << (63 - sh));
}

// Bits 2j of x packed into bit j.
__host__ __device__ __forceinline__ u32 even_bits(u64 x) {
  u32 lo = (u32)x & 0x55555555u, hi = (u32)(x >> 32) & 0x55555555u;
  lo = (lo | (lo >> 1)) & 0x33333333u;
  hi = (hi | (hi >> 1)) & 0x33333333u;
  lo = (lo | (lo >> 2)) & 0x0f0f0f0fu;
  hi = (hi | (hi >> 2)) & 0x0f0f0f0fu;
  lo = (lo | (lo >> 4)) & 0x00ff00ffu;
  hi = (hi | (hi >> 4)) & 0x00ff00ffu;
  lo = (lo | (lo >> 8)) & 0x0000ffffu;
  hi = (hi | (hi >> 8)) & 0x0000ffffu;
  return lo | (hi << 16);
}

// The low and the high bits of the 32 bases from base g of a read on (base g topmost).
__device__ __forceinline__ uint2 load_planes(const uint2 *p, int g) {
  const uint2 a = __ldg(p + (g >> 5)), b = __ldg(p + (g >> 5) + 1);
  return make_uint2(__funnelshift_l(b.x, a.x, g), __funnelshift_l(b.y, a.y, g));
}

// m without the bits of bases that are N in A (from ga) or T (from gt).
__device__ __forceinline__ u32 drop_n(u32 m, const u64 *An, int ga, const u64 *Tn, int gt) {
  if (An) m &= ~__brev(even_bits(load_win32(An, ga)));
  if (Tn) m &= ~__brev(even_bits(load_win32(Tn, gt)));
  return m;
}

// Number of leading bases (0..32) that agree between A (from a) and T (from t), an N
// matching anything (prefixEditDistance-forward.C:164).  An extension to the left
// (-reverse.C:186) compares the reads' reverse complements.
__device__ __forceinline__ int match_run32(const SeqView &A, int a, const SeqView &T, int t) {
  const uint2 x = load_planes(A.p, a), y = load_planes(T.p, t);
  u32         m = (x.x ^ y.x) | (x.y ^ y.y);
  if (A.nm || T.nm) m = drop_n(m, A.nm, a, T.nm, t);
  return __clz((int)m);
}

__device__ __forceinline__ u64 mix64(u64 x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return x;
}

// K-mer table (device): open addressing over 16-byte slots, slot s = (key kv[2s],
// value kv[2s+1]) so that a probe is one 16-byte load.  value: bits 0-31 first
// occurrence, 32-62 count, 63 screened.
struct TableDev {
  const u64 *kv;
  u64        mask;       // capacity - 1
  const u64 *occ;        // (blockString << 32) | offset, ascending within a k-mer
  const unsigned char *lscr, *rscr;   // String_Info l/rfrag_end_screened per block string
  const u32 *slen;       // per block string: length (0 when the string is empty)
  const u32 *sread;      // per block string: 0-based read index
  u32        firstID;    // Hash_String_Num_Offset
  u32        nStrings;
};

__device__ __forceinline__ bool table_find(const TableDev &T, u64 key, u64 &val) {
  u64 s = mix64(key) & T.mask;
  for (u64 probe = 0; probe <= T.mask; probe++) {
    const ulonglong2 e = __ldg((const ulonglong2 *)T.kv + s);
    if (e.x == key) {
      val = e.y;
      return true;
    }
    if (e.x == kEmptyKey) return false;
    s = (s + 1) & T.mask;
  }
  return false;
}

// Parameters every kernel needs (passed by value).
struct DevParams {
  double maxErate;
  double branchMatchValue;     // prefixEditDistance.C:86
  double minBranchTailSlope;   // prefixEditDistance.C:29
  double kmerExpect;           // exp(-K * maxErate), host glibc
  unsigned long long minKmers; // Filter_By_Kmer_Count after overlapInCore.C:410-411 (0 = off)
  int    kmerLen;
  int    partial;
  int    unique;
  int    hopeless;
  int    minOlapLen;
  int    maxErrors;            // MAX_ERRORS (prefixEditDistance.C:27)
  int    collect;              // pairs are collected
  int    pad;
};

__device__ __forceinline__ int error_bound(int i, double maxErate) {
  return (int)ceil(__dmul_rn((double)i, maxErate));   // prefixEditDistance.C:60
}

// The sum of v over the warp, in every lane.
__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace oic

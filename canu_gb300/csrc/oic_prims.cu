// oic_prims.cu -- exclusive scan and stable LSD radix sort (hand-written, no library).
//
// Scan: three-phase (per-tile reduce, recursive scan of tile sums, per-tile scan).
// Sort: 8-bit digits; per pass an upsweep histogram per 4096-key tile (digit-major,
// so one exclusive scan gives every (digit, tile) its output base), then a downsweep
// that ranks keys stably inside the tile, groups the tile by digit in shared memory and
// writes each digit's run out with coalesced stores.
#include "oic_prims.cuh"

namespace oic {

thread_local unsigned long long g_launches = 0;

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems   = 16;
constexpr int kScanTile    = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix and
// sets blockTotal (same value in every thread).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t &blockTotal) {
  constexpr int NW = kScanThreads / 32;
  __shared__ uint32_t warpSums[NW + 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = warp_incl_scan(v);
  if (lane == 31) warpSums[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t s  = (lane < NW) ? warpSums[lane] : 0;
    uint32_t si = warp_incl_scan(s);
    if (lane < NW) warpSums[lane] = si - s;
    if (lane == NW - 1) warpSums[NW] = si;
  }
  __syncthreads();
  blockTotal = warpSums[NW];
  uint32_t r = warpSums[wid] + incl - v;
  __syncthreads();
  return r;
}

// A launch whose element count is only known on the device is sized for a capacity n: it has
// this many blocks at most, which take the tiles that are there in turn, and costs what the
// count costs, not what the capacity does.  (With a block per tile of the capacity, 32 M
// pairs, the sort, the scan and the copy around the DP of 660 pairs took 0.7 ms.)
constexpr unsigned kDevBlocks = 1216;

unsigned tile_blocks(uint64_t tiles, const uint32_t *nDev) {
  return (unsigned)(nDev && tiles > kDevBlocks ? kDevBlocks : tiles);
}

// The elements of a scan: n, or as many as the device's count makes -- the sums of `level`
// scans' tiles over *dev entries, or over the digit counts of *dev keys' sort tiles.
struct ScanCount {
  uint64_t        n;
  const uint32_t *dev;
  uint32_t        keysPerTile;   // of the sort, 256 counts each; 0: entries
  int             level;
  __device__ uint64_t get() const {
    if (!dev) return n;
    uint64_t x = *dev;
    if (keysPerTile) x = (x + keysPerTile - 1) / keysPerTile * 256;
    for (int l = 0; l < level; l++) x = (x + kScanTile - 1) / kScanTile;
    return x < n ? x : n;
  }
};

__global__ void scan_reduce_kernel(const uint32_t *in, ScanCount count, uint32_t *blockSums) {
  const uint64_t n = count.get();
  for (uint64_t tile = blockIdx.x; tile * kScanTile < n; tile += gridDim.x) {
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      uint64_t i = tile * kScanTile + (uint64_t)k * kScanThreads + threadIdx.x;
      if (i < n) s += in[i];
    }
    uint32_t tot;
    block_excl_scan(s, tot);
    if (threadIdx.x == 0) blockSums[tile] = tot;
  }
}

__global__ void scan_tile_kernel(const uint32_t *in, uint32_t *out, ScanCount count, const uint32_t *blockOffsets,
                                 uint32_t *total) {
  const uint64_t n = count.get();
  if (total && n == 0 && threadIdx.x == 0) *total = 0;
  for (uint64_t tile = blockIdx.x; tile * kScanTile < n; tile += gridDim.x) {
    const uint64_t base = tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      uint64_t i = base + k;
      v[k]       = (i < n) ? in[i] : 0;
      s += v[k];
    }
    uint32_t tot;
    uint32_t pre = block_excl_scan(s, tot);
    uint32_t off = (blockOffsets ? blockOffsets[tile] : 0) + pre;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      uint64_t i = base + k;
      if (i < n) out[i] = off;
      off += v[k];
    }
    if (total && threadIdx.x == 0) *total = tot;   // one tile
  }
}

cudaError_t scan_levels(const uint32_t *in, uint32_t *out, ScanCount count, uint32_t *total, void *scratch,
                        cudaStream_t st) {
  const uint64_t nb = (count.n + kScanTile - 1) / kScanTile;
  if (nb == 1) {
    scan_tile_kernel<<<1, kScanThreads, 0, st>>>(in, out, count, nullptr, total);
    g_launches++;
    return cudaGetLastError();
  }
  uint32_t *sums = (uint32_t *)scratch;
  size_t    here = ((nb * sizeof(uint32_t)) + 255) & ~(size_t)255;
  const unsigned blocks = tile_blocks(nb, count.dev);
  scan_reduce_kernel<<<blocks, kScanThreads, 0, st>>>(in, count, sums);
  g_launches++;
  ScanCount up = count;
  up.n         = nb;
  up.level++;
  cudaError_t e = scan_levels(sums, sums, up, total, (char *)scratch + here, st);
  if (e != cudaSuccess) return e;
  // The recursive call scans `sums` in place into block offsets.
  scan_tile_kernel<<<blocks, kScanThreads, 0, st>>>(in, out, count, sums, nullptr);
  g_launches++;
  return cudaGetLastError();
}

}  // namespace

size_t scan_u32_scratch(uint64_t n) {
  uint64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb <= 1) return 0;
  size_t here = ((nb * sizeof(uint32_t)) + 255) & ~(size_t)255;
  return here + scan_u32_scratch(nb);
}

cudaError_t scan_u32(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total, void *scratch, cudaStream_t st,
                     const uint32_t *nDev) {
  if (n == 0) {
    if (total) return cudaMemsetAsync(total, 0, sizeof(uint32_t), st);
    return cudaSuccess;
  }
  return scan_levels(in, out, ScanCount{n, nDev, 0, 0}, total, scratch, st);
}

// ------------------------------------------------------------------------------------
// Radix sort.

namespace {

constexpr int kUpThreads   = 256;                         // upsweep
constexpr int kUpItems     = 16;
constexpr int kSortThreads = 512;                         // downsweep
constexpr int kSortWarps   = kSortThreads / 32;
constexpr int kSortItems   = 8;
constexpr int kSortCtas    = 2;                           // per SM
constexpr int kSortTile    = kSortThreads * kSortItems;   // 4096
constexpr int kDigits      = 256;
static_assert(kUpThreads * kUpItems == kSortTile && kUpThreads == kDigits, "one histogram per downsweep tile");

__global__ void __launch_bounds__(kUpThreads) radix_upsweep_kernel(const unsigned long long *keys, uint64_t n, int shift,
                                                                     uint32_t *hist, const uint32_t *nDev) {
  __shared__ uint32_t h[(kUpThreads / 32)][kDigits];
  if (nDev && *nDev < n) n = *nDev;
  const uint32_t nTiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  const int wid = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
    const uint64_t base = (uint64_t)tile * kSortTile;
    for (int i = threadIdx.x; i < (kUpThreads / 32) * kDigits; i += kUpThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    // All of a thread's loads in flight before the first count: 62 M keys in 76 us (6.6 TB/s;
    // four at a time 128 us).
    unsigned long long k[kUpItems];
#pragma unroll
    for (int it = 0; it < kUpItems; it++) {
      const uint64_t i = base + (uint64_t)it * kUpThreads + threadIdx.x;
      k[it] = i < n ? keys[i] : 0;
    }
#pragma unroll
    for (int it = 0; it < kUpItems; it++)
      if (base + (uint64_t)it * kUpThreads + threadIdx.x < n) atomicAdd(&h[wid][(uint32_t)(k[it] >> shift) & 0xff], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kUpThreads) {
      uint32_t s = 0;
#pragma unroll
      for (int w = 0; w < (kUpThreads / 32); w++) s += h[w][d];
      hist[(uint64_t)d * nTiles + tile] = s;
    }
    __syncthreads();
  }
}

// Downsweep of one 4096-key tile: rank every key inside the tile (stable: warp order,
// then item order, then lane order), place the tile in shared memory grouped by digit, then
// write each digit's run to its output range -- the writes of consecutive threads go to
// consecutive addresses.  VALS false: keys only.
//
// The lanes with the same digit are found with eight ballots: match_any walks a warp's
// distinct digits one by one, and 8 warps x 16 keys of them waited for it two thirds of the
// time (97 G keys/s); marking the lanes in a word per digit in shared memory is as fast as
// the ballots.  62 M keys and values took 385 us (161 G keys/s, 3.8 TB/s) while the tile's
// output ranges were read between two barriers and 8 warps went over the counts twice; read
// ahead, and with two digits to a word, 348 us.  More CTAs on an SM are slower, not faster
// (3 with 40 registers, or tiles of 3,072: +7 %): the output's lines, of 256 runs per tile
// in flight, are what L2 has to hold.
template <bool VALS>
__global__ void __launch_bounds__(kSortThreads, kSortCtas)
    radix_downsweep_kernel(const unsigned long long *keysIn, const uint32_t *valsIn, unsigned long long *keysOut,
                           uint32_t *valsOut, uint64_t n, int shift, const uint32_t *offsets, const uint32_t *nDev) {
  extern __shared__ __align__(16) unsigned char sortDyn[];
  unsigned long long *sk = (unsigned long long *)sortDyn;           // kSortTile keys
  uint32_t           *sv = (uint32_t *)(sk + kSortTile);             // kSortTile values
  __shared__ __align__(4) uint16_t cnt[kSortWarps][kDigits];
  __shared__ uint32_t tileBase[kDigits];     // output position of the tile's first key of each digit ...
  __shared__ uint32_t warpSums[kDigits / 64];
  if (nDev && *nDev < n) n = *nDev;
  const uint32_t nTiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
    const uint64_t tile0 = (uint64_t)tile * kSortTile;
    const uint32_t tot = (uint32_t)(n - tile0 < kSortTile ? n - tile0 : kSortTile);   // the tile's keys
    const uint32_t l0  = (uint32_t)wid * (32 * kSortItems) + lane;                    // this thread's first
    const unsigned ltMask = (1u << lane) - 1;
    unsigned long long k[kSortItems];
    uint32_t v[kSortItems];
    uint32_t rank[kSortItems / 2];             // two 16-bit ranks to a word
#pragma unroll
    for (int it = 0; it < kSortItems; it++) {
      const bool ok = l0 + it * 32 < tot;
      k[it] = ok ? keysIn[tile0 + l0 + it * 32] : 0;
      if (VALS) v[it] = ok ? valsIn[tile0 + l0 + it * 32] : 0;
    }
    // Digits 2 t and 2 t + 1 are thread t's; their output ranges come while the keys are ranked.
    const int t = threadIdx.x;
    uint32_t out0 = 0, out1 = 0;
    if (t < kDigits / 2) {
      out0 = offsets[(uint64_t)(2 * t) * nTiles + tile];
      out1 = offsets[(uint64_t)(2 * t + 1) * nTiles + tile];
    }
    for (int i = lane; i < kDigits / 2; i += 32) ((uint32_t *)cnt[wid])[i] = 0;
    __syncwarp();
#pragma unroll
    for (int it = 0; it < kSortItems; it++) {
      const bool ok = l0 + it * 32 < tot;
      const uint32_t d = (uint32_t)(k[it] >> shift) & 0xff;
      unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
      for (int b = 0; b < 8; b++) {
        const bool bit = (d & (1u << b)) != 0;
        const unsigned m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
      }
      const uint32_t c = cnt[wid][d], below = (uint32_t)__popc(peers & ltMask);
      if (it & 1) rank[it / 2] |= (c + below) << 16;
      else rank[it / 2] = c + below;
      __syncwarp();
      if (ok && below == 0) cnt[wid][d] = (uint16_t)(c + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // Per digit: the warps' exclusive prefix and the digit's start inside the tile, for two
    // digits in one word (no half passes 4,096).
    uint32_t s = 0, incl = 0;
    if (t < kDigits / 2) {
#pragma unroll
      for (int w = 0; w < kSortWarps; w++) s += ((uint32_t *)cnt[w])[t];
      incl = warp_incl_scan((s & 0xffff) + (s >> 16));
      if (lane == 31) warpSums[wid] = incl;
    }
    __syncthreads();
    if (t < kDigits / 2) {
      uint32_t start = incl - (s & 0xffff) - (s >> 16);
      for (int w = 0; w < wid; w++) start += warpSums[w];
      const uint32_t next = start + (s & 0xffff);
      uint32_t at = start | next << 16;
#pragma unroll
      for (int w = 0; w < kSortWarps; w++) {
        const uint32_t c = ((uint32_t *)cnt[w])[t];
        ((uint32_t *)cnt[w])[t] = at;
        at += c;
      }
      tileBase[2 * t]     = out0 - start;       // ... minus its place in the tile
      tileBase[2 * t + 1] = out1 - next;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortItems; it++) {
      if (l0 + it * 32 < tot) {
        const uint32_t p = cnt[wid][(uint32_t)(k[it] >> shift) & 0xff] + ((rank[it / 2] >> (16 * (it & 1))) & 0xffff);
        sk[p] = k[it];
        if (VALS) sv[p] = v[it];
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortItems; it++) {
      const uint32_t p = it * kSortThreads + threadIdx.x;
      if (p < tot) {
        const unsigned long long key = sk[p];
        const uint32_t pos = tileBase[(uint32_t)(key >> shift) & 0xff] + p;
        keysOut[pos] = key;
        if (VALS) valsOut[pos] = sv[p];
      }
    }
    __syncthreads();
  }
}

constexpr size_t kDownsweepKeys = (size_t)kSortTile * sizeof(unsigned long long);
constexpr size_t kDownsweepDyn  = kDownsweepKeys + (size_t)kSortTile * sizeof(uint32_t);

}  // namespace

size_t radix_sort_scratch(uint64_t n) {
  uint64_t nTiles = (n + kSortTile - 1) / kSortTile;
  uint64_t nh     = nTiles * kDigits;
  size_t   here   = ((nh * sizeof(uint32_t)) + 255) & ~(size_t)255;
  return here + scan_u32_scratch(nh);
}

cudaError_t radix_sort_u64_u32(unsigned long long *keys, uint32_t *vals, unsigned long long *keysAlt, uint32_t *valsAlt, uint64_t n,
                               int bits, void *scratch, cudaStream_t st, const uint32_t *nDev) {
  if (n <= 1 || bits <= 0) return cudaSuccess;
  uint64_t  nTiles = (n + kSortTile - 1) / kSortTile;
  uint64_t  nh     = nTiles * kDigits;
  uint32_t *hist   = (uint32_t *)scratch;
  void     *scanSc = (char *)scratch + (((nh * sizeof(uint32_t)) + 255) & ~(size_t)255);
  unsigned long long *ks = keys, *kd = keysAlt;
  uint32_t *vs = vals, *vd = valsAlt;
  int       passes = 0;
  const unsigned blocks = tile_blocks(nTiles, nDev);
  const size_t dyn = vals ? kDownsweepDyn : kDownsweepKeys;
  auto down        = vals ? radix_downsweep_kernel<true> : radix_downsweep_kernel<false>;
  cudaError_t e    = cudaFuncSetAttribute(down, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  if (e != cudaSuccess) return e;
  for (int shift = 0; shift < bits; shift += 8, passes++) {
    radix_upsweep_kernel<<<blocks, kUpThreads, 0, st>>>(ks, n, shift, hist, nDev);
    g_launches++;
    e = scan_levels(hist, hist, ScanCount{nh, nDev, kSortTile, 0}, nullptr, scanSc, st);
    if (e != cudaSuccess) return e;
    down<<<blocks, kSortThreads, dyn, st>>>(ks, vs, kd, vd, n, shift, hist, nDev);
    g_launches++;
    unsigned long long *tk = ks; ks = kd; kd = tk;
    uint32_t *tv = vs; vs = vd; vd = tv;
  }
  if (ks != keys) {
    cudaMemcpyAsync(keys, ks, n * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st);
    if (vals) cudaMemcpyAsync(vals, vs, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
  }
  return cudaGetLastError();
}

}  // namespace oic

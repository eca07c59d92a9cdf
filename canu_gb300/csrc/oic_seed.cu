// oic_seed.cu -- seed lookup and per-read-pair match lists, one CTA per (ref read, strand).
//
// Reference: Find_Overlaps (overlapInCore-Find_Overlaps.C:234-336) walks the ref read's
// k-mers in order, looks each one up, and for every occurrence in a read with a larger
// ID calls Add_Ref (:104-163), which appends the seed to that read pair's match list
// with Add_Match (:25-96).  The list rules are order dependent (runs extend only when
// found before the walk stops; move-to-front), so a pair must see its seeds in exactly
// the reference order: ref offsets ascending, and for one offset the occurrences newest
// first.
//
// Here a CTA takes a strand, 256 k-mer offsets at a time (one lookup per thread), and lays
// their occurrences out as seeds in shared memory, kSeedBuf at a time: stably split by the
// warp that owns the partner read, in reference order within a warp's part.  Each warp
// replays its part 32 seeds per round: the lanes are grouped by partner with match_any, and
// the lowest lane of each group replays its group's seeds in lane order, seeds that follow
// one another on one diagonal in one step.  Different partners advance in parallel; one
// partner's seeds stay in order.  The pair table and node pool
// live in the CTA's HBM scratch; a warp finds the partners it has seen lately in a small
// shared-memory table, and a lane keeps its pair's newest run in registers.
//
// A buffer meets two barriers: one when its owners are counted (by then every warp has
// replayed the seeds before), one when its seeds are in place.  A warp lays out consecutive
// chunks of 32 seeds, so that the counts are 8 x 8 and each warp scans them for itself, and
// it finds the offsets of 32 consecutive seeds with one vote: the ends of the next 32
// offsets, which are all different, as bits of a word.
//
// What bounds it is latency: a lookup, its occurrences, the pair, its newest run, one after
// another, and the warps of a CTA waiting for the slowest (two fifths of the stall cycles).
// A strand on one warp took 11 ms for 8 kb and 25 ms for 15 kb, whatever else ran; eight
// warps and one step per run of seeds bring that to 4 and 7 ms.  With many strands
// (150 Mbp, 1.8 G seeds) the stage went from 53 ms (a warp per strand) to 46 and, with two
// barriers per buffer in place of five, the vote in place of a search per seed, and a
// binary search in place of a scan of the occurrences, to 36.5 ms, of which 26 are the
// lookups and the laying out.  760 to 1,216 strands in flight keep their pairs and runs in
// L2 where 4,864 did not.  5 / 6 / 7 / 8 CTAs per SM: 43.7 / 40.3 / 38.8 / 36.5 ms; a
// buffer of 512 seeds 38.3.  Seeds one by one in the lane loop: 122 ms (of 46).  Fetching
// the next offsets' table slots ahead of the replay: 39.6.  Dealing partners to the warps in
// order of appearance instead of by hash changed less than the spread.
//
// A table probe is one 16-byte load of a (key, value) slot.  The qualifying
// occurrences of a k-mer (partner ID above the ref read's) are the tail of its run,
// which ascends by partner.
#include "oic_kernels.cuh"
#include "oic_occurrences.h"
#include "oic_prims.cuh"

namespace oic {

namespace {

// The block string of occurrence p (the high half of its word).
struct OccStr {
  const u64 *occ;
  __device__ __forceinline__ u32 operator()(u32 p) const { return __ldg((const u32 *)occ + 2 * (u64)p + 1); }
};

constexpr int kSeedThreads = 256;
constexpr int kSeedCtas    = 8;      // CTAs per SM
constexpr int kSeedWarps   = kSeedThreads / 32;
constexpr int kSeedBuf     = 1024;   // seeds laid out at a time
constexpr int kSeedPer     = kSeedBuf / kSeedThreads;   // 32-seed chunks a warp lays out
static_assert(kSeedWarps == 8 && 32 * kSeedPer <= 256, "owners have three bits, ranks a byte");
constexpr int kOffBits     = 24;     // a packed seed: the ref offset above its 256, the partner's offset below
static_assert((u64)kSeedThreads * kSeedNodeCapMax <= 1ull << 32, "the seeds of kSeedThreads offsets are counted in 32 bits");
static_assert(kSeedThreads <= 256 && kMaxReadLenBits <= kOffBits, "both offsets share a word");
constexpr int kSeedRecent  = 64;     // recently seen partners per warp

struct SeedSmem {
  u64 recent[kSeedWarps][kSeedRecent];   // partner << 32 | pair index (all ones: none)
  u32 tStr[kSeedBuf];                    // the seeds: partner, packed offsets
  u32 off[kSeedBuf];
  // The offsets with seeds, in order: seeds up to and with this offset, the place of its seed 0
  // in the occurrence array plus the seeds before it, and the offset.
  u32 end[kSeedThreads];
  u32 from[kSeedThreads];
  unsigned char at[kSeedThreads];
  u32 cnt[kSeedWarps][kSeedWarps / 2];   // seeds per owner and laying warp, two warps to a word
  u32 warpSum[2][kSeedWarps];
  u32 warpCnt[2][kSeedWarps];
  int tooMany[2];                        // one of these offsets has more seeds than there are nodes
  u32 seg;
  u32 base[2];                           // output places of the strand's nodes and pairs
  int nPairs, nNodes, overflow, screened;
};

__device__ __forceinline__ u32 warp_incl_scan_u32(u32 v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    u32 t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Add_Match (Find_Overlaps.C:25-96) on the node pool; head is the pair's list head.
__device__ __forceinline__ bool add_match(int4 *nodes, SeedSmem &sm, int nodeCap, int &head, int tOff, int sOff,
                                          int &consistent, int K) {
  int diag = 0, expected = 0, checked = 0;
  const int newDiag = tOff - sOff;
  bool mtf = false;
  int  link = -1;   // -1: the list head; otherwise the node whose .w (next) links `cur`
  int  cur  = head;
  while (cur != 0) {
    int4 nd  = nodes[cur];   // x offset, y len, z start, w next
    expected = nd.z + nd.y - K + 1;
    diag     = nd.x - nd.z;
    if (expected < sOff) break;
    if (expected == sOff) {
      if (newDiag == diag) {
        nodes[cur].y = nd.y + 1;
        if (mtf) {
          // unlink cur (its predecessor exists because mtf was set on an earlier node)
          nodes[link].w = nd.w;
          nodes[cur].w  = head;
          head          = cur;
        }
        return true;
      } else
        mtf = true;
    }
    checked++;
    link = cur;
    cur  = nd.w;
  }
  if (head != 0 && (checked > 0 || abs(diag - newDiag) > 3 || sOff < expected + K - 2)) consistent = 0;
  int id = atomicAdd(&sm.nNodes, 1);
  if (id >= nodeCap) {
    sm.overflow = 1;
    return false;
  }
  nodes[id] = make_int4(tOff, K, sOff, head);
  head      = id;
  return true;
}

// Inclusive scan over the CTA's threads; `total` is the sum.
__device__ __forceinline__ u32 block_incl_scan(SeedSmem &sm, u32 v, u32 &total) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u32 inc = warp_incl_scan_u32(v);
  __syncthreads();
  if (lane == 31) sm.warpSum[0][wib] = inc;
  __syncthreads();
  u32 before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kSeedWarps; w++) {
    const u32 x = sm.warpSum[0][w];
    before += w < wib ? x : 0;
    all += x;
  }
  total = all;
  return before + inc;
}

// Replays the seeds of one round (lane's seed at place `at` of the buffer, -1: none).
__device__ __forceinline__ void replay_round(SeedSmem &sm, const SeedCaps &cap, int *slotKey, int *slotVal,
                                             PairAcc *pairs, int4 *nodes, int at, int i0, int K) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u32 tStr = at >= 0 ? sm.tStr[at] : (0x80000000u | lane);
  const u32 off  = at >= 0 ? sm.off[at] : 0;
  const unsigned peers = __match_any_sync(0xffffffffu, tStr);
  // Seeds that follow their predecessor in the group: next offset, same diagonal.
  const unsigned before = peers & ((1u << lane) - 1);
  const int      pl = before ? 31 - __clz((int)before) : lane;
  const u32      po = __shfl_sync(0xffffffffu, off, pl);
  const unsigned follows = __ballot_sync(0xffffffffu, before && off == po + (1u << kOffBits) + 1);
  const int  at0  = at - lane;   // lane 0's place: the round's seeds are consecutive
  const bool lead = at >= 0 && before == 0 && !*(volatile int *)&sm.overflow;
  if (lead) {
    // Find or create the pair (Add_Ref, Find_Overlaps.C:104-150).
    u32 h = tStr * 0x9e3779b1u;
    h ^= h >> 15;
    u64 &rec    = sm.recent[wib][(h >> 4) & (kSeedRecent - 1)];
    const u64 r = rec;
    int pi      = (u32)(r >> 32) == tStr ? (int)(u32)r : -1;
    if (pi < 0) {
      int slot = (int)(h & (u32)(cap.slotCap - 1));
      for (int probe = 0; probe < cap.slotCap; probe++) {
        const int old = atomicCAS(&slotKey[slot], -1, (int)tStr);
        if (old == -1) {
          pi = atomicAdd(&sm.nPairs, 1);
          if (pi >= cap.pairCap) {
            pi = -1;
            break;
          }
          PairAcc &pa   = pairs[pi];
          pa.T          = tStr;
          pa.head       = 0;
          pa.diagCt     = 0;
          pa.diagBgn    = (int)kMaxReadLen;
          pa.diagEnd    = 0;
          pa.consistent = 1;
          pa.slot       = slot;
          slotVal[slot] = pi;
          break;
        }
        if (old == (int)tStr) {
          pi = slotVal[slot];
          break;
        }
        slot = (slot + 1) & (cap.slotCap - 1);
      }
      if (pi >= 0) rec = ((u64)tStr << 32) | (u32)pi;
    }
    if (pi < 0) sm.overflow = 1;
    else {
      int4 *const acc = (int4 *)(pairs + pi);
      const int4 a0 = *acc;
      int  head = a0.x, diagCt = a0.y, diagBgn = a0.z, diagEnd = a0.w, consistent = 1;
      int4 hd   = make_int4(0, 0, 0, 0);    // the newest run, and whether it has grown here
      bool dirty = false;
      if (head) hd = nodes[head];
      unsigned m = peers;
      while (m) {
        const int q    = __ffs((int)m) - 1;
        const u32 o    = sm.off[at0 + q];
        const int sOff = i0 + (int)(o >> kOffBits), tOff = (int)(o & ((1u << kOffBits) - 1));
        // Seed q, and the `more` seeds of the group that follow it one by one.
        const unsigned brk = m & ~follows & ~((2u << q) - 1);
        const unsigned run = brk ? m & ((brk & (0u - brk)) - 1) : m;
        int more = __popc(run) - 1;
        m &= m - 1;
        diagCt++;
        if (diagBgn > sOff) diagBgn = sOff;
        if (diagEnd < sOff) diagEnd = sOff;
        // Add_Match's first node (Find_Overlaps.C:25-96): most seeds extend it.
        const int expected = hd.z + hd.y - K + 1, diag = hd.x - hd.z, newDiag = tOff - sOff;
        if (head && expected >= sOff) {
          if (expected == sOff && newDiag == diag) {
            hd.y++;
            dirty = true;
          } else {
            if (dirty) nodes[head].y = hd.y;
            dirty = false;
            if (!add_match(nodes, sm, cap.nodeCap, head, tOff, sOff, consistent, K)) break;
            hd = nodes[head];
            // Unless the seed's run is now the first node, the next seed walks the list too.
            if (hd.z + hd.y - K != sOff || hd.x - hd.z != newDiag) more = 0;
          }
        } else {
          // The walk stops at the first node: a new run.
          if (head && (abs(diag - newDiag) > 3 || sOff < expected + K - 2)) consistent = 0;
          const int id = atomicAdd(&sm.nNodes, 1);
          if (id >= cap.nodeCap) {
            sm.overflow = 1;
            break;
          }
          if (dirty) nodes[head].y = hd.y;
          dirty     = false;
          hd        = make_int4(tOff, K, sOff, head);
          nodes[id] = hd;
          head   = id;
        }
        if (more) {
          // Each of them extends the first node by one.
          hd.y += more;
          dirty = true;
          diagCt += more;
          if (diagEnd < sOff + more) diagEnd = sOff + more;
          m &= ~run;
        }
      }
      if (dirty) nodes[head].y = hd.y;
      *acc = make_int4(head, diagCt, diagBgn, diagEnd);
      if (!consistent) pairs[pi].consistent = 0;
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kSeedThreads, kSeedCtas) seed_kernel(ReadsDev R, TableDev T, DevParams P, const u32 *segReads,
                                                               const u32 *segList, u32 nSeg, u32 *segCounter,
                                                               SeedScratch sc, SeedCaps cap, SeedOut out) {
  __shared__ SeedSmem sm;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  int     *slotKey = sc.slotKey + (u64)blockIdx.x * cap.slotCap;
  int     *slotVal = sc.slotVal + (u64)blockIdx.x * cap.slotCap;
  PairAcc *pairs   = sc.pairs + (u64)blockIdx.x * cap.pairCap;
  int4    *nodes   = sc.nodes + (u64)blockIdx.x * cap.nodeCap;
  const int K      = P.kmerLen;
  const u64 kmask  = (K >= 32) ? ~0ull : ((1ull << (2 * K)) - 1);
  unsigned long long nSeeds = 0, nSegs = 0;
  int par = 0;   // which half of warpSum and warpCnt the next 256 offsets take

  for (int i = tid; i < cap.slotCap; i += kSeedThreads) slotKey[i] = -1;

  while (true) {
    __syncthreads();
    if (tid == 0) {
      sm.seg      = atomicAdd(segCounter, 1u);
      sm.nPairs   = 0;
      sm.nNodes   = 1;
      sm.overflow = 0;
      sm.screened = 0;
      sm.tooMany[0] = sm.tooMany[1] = 0;
    }
    for (int i = tid; i < kSeedWarps * kSeedRecent; i += kSeedThreads) (&sm.recent[0][0])[i] = ~0ull;
    __syncthreads();
    if (sm.seg >= nSeg) break;
    const u32 seg = segList ? segList[sm.seg] : sm.seg;   // segment = (ref index << 1) | strand
    nSegs++;

    const u32 sRead = segReads[seg >> 1];
    const int dir   = seg & 1;
    const u64 wo    = R.wordOff[sRead];
    const u64 *Sw   = (dir ? R.rc : R.fwd) + wo;
    const u64 *Sn   = R.hasN[sRead] ? (dir ? R.nrc : R.nfwd) + wo : nullptr;
    const int sLen  = (int)R.len[sRead];
    const int nK    = sLen - K + 1;
    // A partner qualifies from this string on.
    const u32 from = sRead + 2 > T.firstID ? sRead + 2 - T.firstID : 0;
    unsigned long long segSeeds = 0;   // counted once the segment completes in this configuration

    for (int i0 = 0; i0 < nK; i0 += kSeedThreads) {
      const int i = i0 + tid;
      u32 n = 0, qEnd = 0;
      if (i < nK) {
        u64 key = load_win32(Sw, i) & kmask;
        bool ok = !(Sn && (load_win32(Sn, i) & kmask));
        u64 val;
        if (ok && table_find(T, key, val)) {
          if (val >> 63) {
            // hi_hits (Find_Overlaps.C:274-276 for offset 0, :310-317 otherwise)
            int scr = 0;
            if (i == 0) scr = 1;
            else {
              if (i < kHopelessMatch) scr = 1;
              if (sLen - i - K + 1 < kHopelessMatch) scr |= 2;
            }
            if (scr) atomicOr(&sm.screened, scr);
          } else {
            // The qualifying occurrences are the run's end: it ascends by partner.
            const u32 start = (u32)(val & 0xffffffffull);
            qEnd            = start + (u32)((val >> 32) & 0x7fffffffull);
            n = offset_seeds(start, qEnd, from, (u32)cap.nodeCap, OccStr{T.occ});
            if (n == kTooManySeeds) {
              n               = 0;
              sm.tooMany[par] = 1;
            }
          }
        }
      }
      // The offsets that have seeds, in order.
      const unsigned has = __ballot_sync(0xffffffffu, n > 0);
      const u32 inc = warp_incl_scan_u32(n);
      if (lane == 31) {
        sm.warpSum[par][wib] = inc;
        sm.warpCnt[par][wib] = __popc(has);
      }
      __syncthreads();
      // Only a replay sets the flag, and none runs between this barrier and the next: all warps
      // read the same.  (So it is after the buffer's counts below.)  tooMany is written before
      // the barrier, its other half before the next one.
      if (sm.overflow | sm.tooMany[par]) break;
      u32 end = inc, total = 0;
      int c = __popc(has & ((1u << lane) - 1)), nOff = 0;
#pragma unroll
      for (int w = 0; w < kSeedWarps; w++) {
        const u32 x = sm.warpSum[par][w], y = sm.warpCnt[par][w];
        end += w < wib ? x : 0;
        c += w < wib ? y : 0;
        total += x;
        nOff += y;
      }
      par ^= 1;
      if (total == 0) continue;
      if (n) {
        sm.end[c]  = end;
        sm.from[c] = qEnd - 1 + (end - n);
        sm.at[c]   = (unsigned char)tid;
      }
      segSeeds += (tid == 0) ? total : 0;
      __syncthreads();

      for (u32 b = 0; b < total; b += kSeedBuf) {
        // Seeds b .. b + kSeedBuf, in reference order; this warp lays out `per` chunks of 32.
        const u32 stop = total - b < (u32)kSeedBuf ? total : b + kSeedBuf;
        const int per  = (int)((stop - b + 32 * kSeedWarps - 1) / (32 * kSeedWarps));
        u32 s0 = b + 32 * per * wib;
        u32 tS[kSeedPer], off[kSeedPer], ranks = 0, run = 0;
        // The first offset with seeds past s0.
        int c0 = 0;
        if (s0 < stop) {
          c0 = 8 * __popc(__ballot_sync(0xffffffffu, 8 * lane + 7 < nOff && sm.end[8 * lane + 7] <= s0));
          c0 += __popc(__ballot_sync(0xffffffffu, lane < 8 && c0 + lane < nOff && sm.end[c0 + lane] <= s0));
        }
#pragma unroll
        for (int k = 0; k < kSeedPer; k++) {
          if (k >= per || s0 >= stop) break;
          // The ends of the next 32 offsets, as bits: seed s0 + l is past those below bit l.
          const u32 d = c0 + lane < nOff ? sm.end[c0 + lane] - s0 : 33;
          const unsigned ends = __reduce_or_sync(0xffffffffu, d <= 32 ? 1u << (d - 1) : 0);
          const int  j  = c0 + __popc(ends & ((1u << lane) - 1));
          const bool ok = s0 + lane < stop;
          tS[k] = off[k] = 0;
          if (ok) {
            const u64 o = __ldg(T.occ + (u32)(sm.from[j] - (s0 + lane)));   // newest occurrence first
            tS[k]  = (u32)(o >> 32);
            off[k] = (u32)sm.at[j] << kOffBits | (u32)o;
          }
          // Its owner, and its rank among the owner's seeds of this warp; lane w counts owner w's.
          const u32 w = (tS[k] * 0x9e3779b1u) >> 29;
          const unsigned v0 = __ballot_sync(0xffffffffu, w & 1), v1 = __ballot_sync(0xffffffffu, w & 2),
                         v2 = __ballot_sync(0xffffffffu, w & 4), in = __ballot_sync(0xffffffffu, ok);
          const unsigned same = (w & 1 ? v0 : ~v0) & (w & 2 ? v1 : ~v1) & (w & 4 ? v2 : ~v2) & in;
          ranks |= (__shfl_sync(0xffffffffu, run, w) + __popc(same & ((1u << lane) - 1))) << (8 * k);
          run += __popc((lane & 1 ? v0 : ~v0) & (lane & 2 ? v1 : ~v1) & (lane & 4 ? v2 : ~v2) & in);
          c0 += __popc(ends);
          s0 += 32;
        }
        if (lane < kSeedWarps) ((unsigned short *)sm.cnt[lane])[wib] = (unsigned short)run;
        __syncthreads();   // every warp has replayed its part of the seeds before these
        if (sm.overflow) break;
        // Places: by owner, then by laying warp.
        const u32 x   = (&sm.cnt[0][0])[lane];
        const u32 sum = (x & 0xffff) + (x >> 16);
        const u32 up  = warp_incl_scan_u32(sum);
        const u32 place = up - sum + (wib & 1 ? x & 0xffff : 0);
        const int first = (int)__shfl_sync(0xffffffffu, up - sum, 4 * wib);
        const int last  = (int)__shfl_sync(0xffffffffu, up, 4 * wib + 3);
        s0 = b + 32 * per * wib;
#pragma unroll
        for (int k = 0; k < kSeedPer; k++) {
          if (k >= per || s0 >= stop) break;
          const u32 w = (tS[k] * 0x9e3779b1u) >> 29;
          const u32 p = __shfl_sync(0xffffffffu, place, 4 * w + (wib >> 1)) + ((ranks >> (8 * k)) & 0xff);
          if (s0 + lane < stop) {
            sm.tStr[p] = tS[k];
            sm.off[p]  = off[k];
          }
          s0 += 32;
        }
        __syncthreads();
        for (int r = first; r < last; r += 32)
          replay_round(sm, cap, slotKey, slotVal, pairs, nodes, r + lane < last ? r + lane : -1, i0, K);
      }
    }
    __syncthreads();
    const int  nPairs = min(sm.nPairs, cap.pairCap);
    const bool ovf    = (sm.overflow | sm.tooMany[0] | sm.tooMany[1]) != 0;
    const bool lscr = sm.screened & 1, rscr = sm.screened & 2;
    if (!ovf) nSeeds += segSeeds;

    if (!ovf && nPairs > 0) {
      // Every run is a node of one pair: sm.nNodes - 1 of them.  One output allocation for
      // the strand.
      const u32 nodeTotal = (u32)(sm.nNodes - 1);
      if (tid == 0) {
        sm.base[0] = atomicAdd(out.nodeCount, nodeTotal);
        sm.base[1] = atomicAdd(out.pairCount, (u32)nPairs);
      }
      __syncthreads();
      const u32 nodeBase = sm.base[0], pairBase = sm.base[1];
      const bool fits = (u64)nodeBase + nodeTotal <= out.nodeCap && (u64)pairBase + nPairs <= out.pairCap;
      if (!fits) {
        if (tid == 0) atomicOr(out.err, kErrOutNodes);
      } else {
        u32 run = nodeBase;
        for (int p0 = 0; p0 < nPairs; p0 += kSeedThreads) {
          const int p = p0 + tid;
          u32 c = 0, all;
          if (p < nPairs)
            for (int q = pairs[p].head; q != 0; q = nodes[q].w) c++;
          const u32 my = run + block_incl_scan(sm, c, all) - c;
          if (p < nPairs) {
            u32 k = my;
            for (int q = pairs[p].head; q != 0;) {
              const int4 nd  = nodes[q];
              out.nodes[k++] = make_int4(nd.x, nd.y, nd.z, 0);
              q              = nd.w;
            }
            PairRec rec;
            rec.sRead   = sRead;
            rec.tStr    = pairs[p].T;
            rec.nodeOff = my;
            rec.nodeCnt = c;
            rec.diagCt  = pairs[p].diagCt;
            rec.diagBgn = pairs[p].diagBgn;
            rec.diagEnd = pairs[p].diagEnd;
            rec.flags   = (u32)dir | ((u32)(pairs[p].consistent != 0) << 1) | ((u32)lscr << 2) | ((u32)rscr << 3);
            out.pairs[pairBase + p] = rec;
          }
          run += all;
        }
      }
    } else if (ovf && tid == 0) {
      u32 k = atomicAdd(out.overflowCount, 1u);
      out.overflowSegs[k] = seg;
    }
    // Reset the slots this segment used (all of them after an overflow, whose
    // abandoned claims are not all recorded in the pair list).
    if (ovf)
      for (int i = tid; i < cap.slotCap; i += kSeedThreads) slotKey[i] = -1;
    else
      for (int p = tid; p < nPairs; p += kSeedThreads) slotKey[pairs[p].slot] = -1;
  }
  if (tid == 0) {
    atomicAdd(&out.stats[0], nSeeds);
    atomicAdd(&out.stats[1], nSegs);
  }
}

}  // namespace

int seed_ctas_per_sm() { return kSeedCtas; }

void launch_seed(ReadsDev R, TableDev T, DevParams P, const u32 *segReads, const u32 *segList, u32 nSeg,
                 u32 *segCounter, SeedScratch sc, SeedCaps cap, int ctas, SeedOut out, cudaStream_t st) {
  if (nSeg == 0) return;
  const u32 blocks = nSeg < (u32)ctas ? nSeg : (u32)ctas;
  seed_kernel<<<blocks, kSeedThreads, 0, st>>>(R, T, P, segReads, segList, nSeg, segCounter, sc, cap, out);
  g_launches++;
}

}  // namespace oic

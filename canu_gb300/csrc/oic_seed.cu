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
// What bounds it is latency: a lookup, its occurrences, the pair, its newest run, one after
// another, and the warps of a CTA waiting for the one with most seeds (half of the stall
// cycles).  A strand on one warp took 11 ms for 8 kb and 25 ms for 15 kb, whatever else ran;
// eight warps and one step per run of seeds bring that to 4 and 7 ms.  With many strands
// (150 Mbp, 1.8 G seeds) the stage went from 53 to 46 ms: 760 to 1,216 strands in flight
// keep their pairs and runs in L2 where 4,864 did not (37 B of HBM per seed, from 55), and
// a seed costs 19 warp instructions.  5 / 6 / 8 CTAs per SM: 53 / 49 / 46 ms.  Seeds one by
// one in the lane loop: 122 ms.  Dealing partners to the warps in order of appearance
// instead of by hash, or laying the seeds out by offset instead of by a search per seed,
// changed less than the spread.
//
// A table probe is one 16-byte load of a (key, value) slot.  The qualifying
// occurrences of a k-mer (partner ID above the ref read's) are the tail of its run,
// which ascends by partner: runs of up to kScanMax entries are counted by a backward
// scan, eight entries per step -- the entries the replay reads next -- and longer runs
// by binary search.
#include "oic_kernels.cuh"
#include "oic_prims.cuh"

namespace oic {

namespace {

constexpr int kSeedThreads = 256;
constexpr int kSeedCtas    = 8;      // CTAs per SM
constexpr int kSeedWarps   = kSeedThreads / 32;
constexpr int kScanMax     = 64;     // occurrence runs up to this long are scanned backwards
constexpr int kSeedBuf     = 1024;   // seeds laid out at a time
constexpr int kSeedPer     = kSeedBuf / kSeedThreads;
constexpr int kSeedChunks  = kSeedBuf / 32;
static_assert(kSeedChunks == 32 && kSeedWarps == 8, "one lane per chunk; owners have three bits");
constexpr int kSeedRecent  = 64;     // recently seen partners per warp

struct SeedSmem {
  u64 recent[kSeedWarps][kSeedRecent];   // partner << 32 | pair index (all ones: none)
  u32 tStr[kSeedBuf];                    // the seeds: partner, its offset, the ref strand's offset
  int tOff[kSeedBuf];
  int sOff[kSeedBuf];
  u32 incl[kSeedThreads];                // inclusive scan of the offsets' seed counts
  u32 qEnd[kSeedThreads];
  unsigned short cnt[kSeedWarps][kSeedChunks];   // seeds of a warp in 32 consecutive ones, then their places
  u32 part[kSeedWarps];                  // seeds of a warp in the buffer
  u32 warpSum[kSeedWarps];
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
  if (lane == 31) sm.warpSum[wib] = inc;
  __syncthreads();
  u32 before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kSeedWarps; w++) {
    const u32 x = sm.warpSum[w];
    before += w < wib ? x : 0;
    all += x;
  }
  total = all;
  return before + inc;
}

// Replays the seeds of one round (lane's seed at place `at` of the buffer, -1: none).
__device__ __forceinline__ void replay_round(SeedSmem &sm, const SeedCaps &cap, int *slotKey, int *slotVal,
                                             PairAcc *pairs, int4 *nodes, int at, int K) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u32 tStr = at >= 0 ? sm.tStr[at] : (0x80000000u | lane);
  const int myS  = at >= 0 ? sm.sOff[at] : 0, myT = at >= 0 ? sm.tOff[at] : 0;
  const unsigned peers = __match_any_sync(0xffffffffu, tStr);
  // Seeds that follow their predecessor in the group: next offset, same diagonal.
  const unsigned before = peers & ((1u << lane) - 1);
  const int      pl = before ? 31 - __clz((int)before) : lane;
  const int      ps = __shfl_sync(0xffffffffu, myS, pl), pt = __shfl_sync(0xffffffffu, myT, pl);
  const unsigned follows = __ballot_sync(0xffffffffu, before && myS == ps + 1 && myT == pt + 1);
  const int  at0  = at - lane;   // lane 0's place: the round's seeds are consecutive
  const bool lead = at >= 0 && before == 0 && !*(volatile int *)&sm.overflow;
  if (lead) {
    // Find or create the pair (Add_Ref, Find_Overlaps.C:104-150).
    const u32 h = (u32)(mix64(tStr));
    u64 &rec    = sm.recent[wib][(h >> 16) & (kSeedRecent - 1)];
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
      PairAcc pa  = pairs[pi];
      int4    hd  = make_int4(0, 0, 0, 0);    // the newest run, and whether it has grown here
      bool    dirty = false;
      if (pa.head) hd = nodes[pa.head];
      unsigned m = peers;
      while (m) {
        const int q    = __ffs((int)m) - 1;
        const int sOff = sm.sOff[at0 + q], tOff = sm.tOff[at0 + q];
        // Seed q, and the `more` seeds of the group that follow it one by one.
        const unsigned brk = m & ~follows & ~((2u << q) - 1);
        const unsigned run = brk ? m & ((brk & (0u - brk)) - 1) : m;
        int more = __popc(run) - 1;
        m &= m - 1;
        pa.diagCt++;
        if (pa.diagBgn > sOff) pa.diagBgn = sOff;
        if (pa.diagEnd < sOff) pa.diagEnd = sOff;
        // Add_Match's first node (Find_Overlaps.C:25-96): most seeds extend it.
        const int expected = hd.z + hd.y - K + 1, diag = hd.x - hd.z, newDiag = tOff - sOff;
        if (pa.head && expected >= sOff) {
          if (expected == sOff && newDiag == diag) {
            hd.y++;
            dirty = true;
          } else {
            if (dirty) nodes[pa.head].y = hd.y;
            dirty = false;
            if (!add_match(nodes, sm, cap.nodeCap, pa.head, tOff, sOff, pa.consistent, K)) break;
            hd = nodes[pa.head];
            // Unless the seed's run is now the first node, the next seed walks the list too.
            if (hd.z + hd.y - K != sOff || hd.x - hd.z != newDiag) more = 0;
          }
        } else {
          // The walk stops at the first node: a new run.
          if (pa.head && (abs(diag - newDiag) > 3 || sOff < expected + K - 2)) pa.consistent = 0;
          const int id = atomicAdd(&sm.nNodes, 1);
          if (id >= cap.nodeCap) {
            sm.overflow = 1;
            break;
          }
          if (dirty) nodes[pa.head].y = hd.y;
          dirty     = false;
          hd        = make_int4(tOff, K, sOff, pa.head);
          nodes[id] = hd;
          pa.head   = id;
        }
        if (more) {
          // Each of them extends the first node by one.
          hd.y += more;
          dirty = true;
          pa.diagCt += more;
          if (pa.diagEnd < sOff + more) pa.diagEnd = sOff + more;
          m &= ~run;
        }
      }
      if (dirty) nodes[pa.head].y = hd.y;
      pairs[pi].head       = pa.head;
      pairs[pi].diagCt     = pa.diagCt;
      pairs[pi].diagBgn    = pa.diagBgn;
      pairs[pi].diagEnd    = pa.diagEnd;
      pairs[pi].consistent = pa.consistent;
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

  for (int i = tid; i < cap.slotCap; i += kSeedThreads) slotKey[i] = -1;

  while (true) {
    __syncthreads();
    if (tid == 0) {
      sm.seg      = atomicAdd(segCounter, 1u);
      sm.nPairs   = 0;
      sm.nNodes   = 1;
      sm.overflow = 0;
      sm.screened = 0;
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
    const i64 thr   = (i64)(sRead + 1) - (i64)T.firstID;   // T qualifies iff tStr > thr
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
            const u32 start = (u32)(val & 0xffffffffull);
            const u32 cnt   = (u32)((val >> 32) & 0x7fffffffull);
            const u32 end   = start + cnt;
            if (cnt <= (u32)kScanMax) {
              while (n < cnt) {
                u64 o[8];
#pragma unroll
                for (int k = 0; k < 8; k++) o[k] = (n + k < cnt) ? __ldg(T.occ + (end - 1 - n - k)) : 0ull;
                u32 q = 0;
#pragma unroll
                for (int k = 0; k < 8; k++)
                  if (q == (u32)k && n + k < cnt && (i64)(o[k] >> 32) > thr) q++;
                n += q;
                if (q < 8) break;
              }
            } else {
              // first occurrence whose string is past thr
              u32 lo = start, hi = end;
              while (lo < hi) {
                u32 mid = (lo + hi) >> 1;
                if ((i64)(T.occ[mid] >> 32) > thr) hi = mid;
                else lo = mid + 1;
              }
              n = end - lo;
            }
            qEnd = end;
          }
        }
      }
      u32 total;
      sm.qEnd[tid] = qEnd;
      sm.incl[tid] = block_incl_scan(sm, n, total);
      segSeeds += (tid == 0) ? total : 0;

      for (u32 b = 0; b < total; b += kSeedBuf) {
        __syncthreads();
        // Seeds b .. b + kSeedBuf, in reference order: thread tid has those at 256 k + tid.
        u32 tS[kSeedPer];
        int tO[kSeedPer], sO[kSeedPer], rank[kSeedPer];
#pragma unroll
        for (int k = 0; k < kSeedPer; k++) {
          const u32  s  = b + kSeedThreads * k + tid;
          const bool ok = s < total;
          tS[k] = 0;
          tO[k] = sO[k] = 0;
          if (ok) {
            int lo = 0, hi = kSeedThreads - 1;   // first offset with incl > s
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if (sm.incl[mid] > s) hi = mid;
              else lo = mid + 1;
            }
            const u32 j = s - (lo ? sm.incl[lo - 1] : 0);
            const u64 o = __ldg(T.occ + (sm.qEnd[lo] - 1 - j));   // newest occurrence first
            tS[k] = (u32)(o >> 32);
            tO[k] = (int)(u32)o;
            sO[k] = i0 + lo;
          }
          // Its owner, and its rank among the owner's seeds of these 32.
          const u32 w = (tS[k] * 0x9e3779b1u) >> 29;
          const unsigned v0 = __ballot_sync(0xffffffffu, w & 1), v1 = __ballot_sync(0xffffffffu, w & 2),
                         v2 = __ballot_sync(0xffffffffu, w & 4), in = __ballot_sync(0xffffffffu, ok);
          const unsigned same = (w & 1 ? v0 : ~v0) & (w & 2 ? v1 : ~v1) & (w & 4 ? v2 : ~v2) & in;
          rank[k] = ok ? __popc(same & ((1u << lane) - 1)) : -1;
          const int chunk = kSeedWarps * k + wib;
          if (lane < kSeedWarps)
            sm.cnt[lane][chunk] = (unsigned short)__popc((lane & 1 ? v0 : ~v0) & (lane & 2 ? v1 : ~v1) &
                                                         (lane & 4 ? v2 : ~v2) & in);
        }
        __syncthreads();
        {
          // Warp w turns its row of counts into places inside its part.
          const u32 c   = sm.cnt[wib][lane];   // kSeedChunks == 32
          const u32 inc = warp_incl_scan_u32(c);
          sm.cnt[wib][lane] = (unsigned short)(inc - c);
          if (lane == 31) sm.part[wib] = inc;
        }
        __syncthreads();
        u32 first = 0;                          // this warp's part of the buffer
        for (int w = 0; w < wib; w++) first += sm.part[w];
        const int mine = (int)sm.part[wib];
#pragma unroll
        for (int k = 0; k < kSeedPer; k++)
          if (rank[k] >= 0) {
            const u32 w = (tS[k] * 0x9e3779b1u) >> 29;
            u32 p = sm.cnt[w][kSeedWarps * k + wib] + rank[k];
            for (u32 x = 0; x < w; x++) p += sm.part[x];
            sm.tStr[p] = tS[k];
            sm.tOff[p] = tO[k];
            sm.sOff[p] = sO[k];
          }
        __syncthreads();
        for (int r = 0; r < mine; r += 32)
          replay_round(sm, cap, slotKey, slotVal, pairs, nodes, r + lane < mine ? (int)first + r + lane : -1, K);
        if (__syncthreads_or(sm.overflow)) break;
      }
      if (__syncthreads_or(sm.overflow)) break;
    }
    __syncthreads();
    const int  nPairs = min(sm.nPairs, cap.pairCap);
    const bool ovf    = sm.overflow != 0;
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

// oic_align.cuh -- warp-cooperative banded prefix edit distance (furthest-reaching
// diagonals) and the per-read-pair driver around it.
//
// One warp owns one read pair.  Lanes own diagonals of the current error row, two each per
// step of 64; the previous row lives in a shared-memory buffer, every kept row is appended to
// the warp's traceback arena in HBM, and the slides compare 32 bases per step on the reads'
// bit planes.  The arithmetic is the reference's exactly -- integer rows, the same band
// pruning against Edit_Match_Limit, the same first-index tie breaks, and the branch-point test in IEEE double with
// explicitly rounded multiply / subtract / divide (no FMA contraction), as an x86-64
// build of canu computes it.
#pragma once

#include "oic_common.cuh"

namespace oic {

// The DP's rows, in dynamic shared memory (each warp its slice from WarpDP::smOff on).
extern __shared__ __align__(16) int smemRows[];

// Per-warp global scratch.
struct WarpScratch {
  int  *arena;       // kept DP rows, band-compacted
  int4 *rowHdr;      // per error row: (arena offset, kept band left, kept band right, unused)
  int  *rowsG;       // two row buffers of rowsGW ints in HBM, used once a band outgrows shared memory
  int  *deltaL;      // Left_Delta (merged delta of the last extension)
  int  *deltaR;      // Right_Delta
  int  *stack;       // Delta_Stack
  unsigned char *alive;   // match-node alive flags of the current pair
};

struct AlignCaps {
  int arenaCap;   // ints per warp
  int rowCap;     // error rows per warp (also bounds the delta arrays)
  int nodeCap;    // match nodes per pair
  int bandW;      // ints per shared-memory row buffer
  int rowsGW;     // ints per HBM row buffer (bands wider than bandW - 4 up to rowsGW - 4)
};

struct WarpDP {
  WarpScratch        sc;
  AlignCaps          cap;
  int               *smA, *smB;     // shared-memory row buffers of a group CTA (bandW ints each)
  int                smOff;         // first int of the warp's slice of smemRows (one-warp rows)
  const int         *eml;           // Edit_Match_Limit
  DevParams          P;
  unsigned long long cells, slides, rows;
  u32                err;           // capacity error of the current pair (0 = ok)
  int                leftLen, rightLen;
  struct GroupShared *gs;           // non-null: warp 0 of a group CTA (row loops on all warps)
  int                gThreads;      // threads of the group CTA
  int                gU;            // diagonals per thread per pass in the group row loop
};

// The scratch of global warp gw inside the base allocations of a configuration.
static __device__ __forceinline__ WarpScratch warp_scratch(const WarpScratch &base, const AlignCaps &cap, u64 gw) {
  WarpScratch s;
  s.arena  = base.arena + gw * (u64)cap.arenaCap;
  s.rowHdr = base.rowHdr + gw * (u64)cap.rowCap;
  s.rowsG  = base.rowsG ? base.rowsG + gw * (u64)(2 * cap.rowsGW) : nullptr;
  s.deltaL = base.deltaL + gw * (u64)(cap.rowCap + 8);
  s.deltaR = base.deltaR + gw * (u64)(cap.rowCap + 8);
  s.stack  = base.stack + gw * (u64)(cap.rowCap + 8);
  s.alive  = base.alive + gw * (u64)cap.nodeCap;
  return s;
}

// Row-0 exact slide shared by the warp: each lane tests one 32-base window per step.
__device__ __forceinline__ int warp_slide0(const SeqView &A, int a0, const SeqView &T, int t0, int m,
                                           unsigned long long &slides) {
  const int lane = threadIdx.x & 31;
  int       run  = m;
  for (int base = 0; base < m; base += 32 * 32) {
    const int off = base + lane * 32;
    const int r   = off < m ? match_run32(A, a0 + off, T, t0 + off) : 32;
    const unsigned stop = __ballot_sync(0xffffffffu, r < 32);
    if (stop) {
      const int f = __ffs((int)stop) - 1;
      run         = min(base + f * 32 + __shfl_sync(0xffffffffu, r, f), m);
      break;
    }
  }
  if (lane == 0) slides += (unsigned long long)run;
  return run;
}

// Traceback of Set_Right_Delta / Set_Left_Delta (prefixEditDistance-forward.C:32-71,
// -reverse.C:36-93) from row e, diagonal d whose value is `last`, by the whole warp (every
// argument and result is warp-uniform).  Writes one entry per indel to out[] (by lane 0;
// a __syncwarp before the caller reads them), their number to nOut; returns the value
// reached on row 0.
//
// A step needs the row above at d - 1, d and d + 1 and moves d by at most one, so the
// values that the next kTraceRows rows can need lie within a window of 32 diagonals: the
// warp loads those windows into its (now unused) shared-memory rows together, one coalesced
// load per row, all in flight, and walks them there.  One lane walking the arena by itself
// waited for an L2 round trip per row.
constexpr int kTraceRows = 12;
static __device__ __noinline__ int trace_rows(const WarpDP &w, int e, int d, int last, int *out, int &nOut) {
  static_assert(kTraceRows + 1 <= 15, "the window holds d - kTraceRows - 1 .. d + kTraceRows + 1");
  const int4 *const rowHdr = w.sc.rowHdr;
  const int *const  arena  = w.sc.arena;
  int *const        tile   = smemRows + w.smOff;
  const int         lane   = threadIdx.x & 31;
  const int4        none   = make_int4(0, 1, 0, 0);   // an empty band
  int  n = 0;
  // Lane j holds the header of row k - 1 - j; the next block's are loaded a block ahead.
  int4 hNext = lane < kTraceRows && e - 1 - lane >= 0 ? rowHdr[e - 1 - lane] : none;
  for (int k = e; k > 0; k -= kTraceRows) {
    const int4 h  = hNext;
    const int  kn = k - kTraceRows - 1 - lane;
    hNext         = lane < kTraceRows && kn >= 0 ? rowHdr[kn] : none;
    const int d0  = d - 16, dd = d0 + lane;
#pragma unroll 6
    for (int j = 0; j < kTraceRows; j++) {
      const int off = __shfl_sync(0xffffffffu, h.x, j), L = __shfl_sync(0xffffffffu, h.y, j),
                R   = __shfl_sync(0xffffffffu, h.z, j);
      tile[32 * j + lane] = (dd >= L && dd <= R) ? arena[off + dd - L] : -2;
    }
    __syncwarp();
    const int rows = min(k, kTraceRows);
#pragma unroll 1
    for (int j = 0; j < rows; j++) {
      const int *g = tile + 32 * j + (d - d0);
      const int g0 = g[0], gm = g[-1], gp = g[1];
      int from = 0, mx = 1 + g0;
      if (gm > mx) { from = -1; mx = gm; }
      if (1 + gp > mx) { from = 1; mx = 1 + gp; }
      if (from) {
        if (lane == 0) out[n] = from < 0 ? mx - last - 1 : last - (mx - 1);
        last = from < 0 ? gm : gp;
        d += from;
        n++;
      }
    }
    __syncwarp();
  }
  nOut = n;
  return last;
}

__device__ __forceinline__ int arena_get(const WarpDP &w, int e, int d) {
  const int4 h = w.sc.rowHdr[e];
  return (d >= h.y && d <= h.z) ? w.sc.arena[h.x + d - h.y] : -2;
}

// Set_Right_Delta (forward.C:32-71) into sc.deltaR, whole warp.
static __device__ __noinline__ void set_right_delta(WarpDP &w, int e, int d, int last) {
  const int  lane  = threadIdx.x & 31;
  int *const stack = w.sc.stack;
  int n;
  const int l = trace_rows(w, e, d, last, stack, n);
  if (lane == 0) stack[n] = l + 1;
  __syncwarp();
  for (int k = lane; k < n; k += 32) {
    const int s      = stack[n - 1 - k];
    w.sc.deltaR[k]   = abs(stack[n - k]) * ((s > 0) - (s < 0));
  }
  w.rightLen = n;
  __syncwarp();
}

// Set_Left_Delta (reverse.C:36-93) into sc.deltaL, whole warp.
static __device__ __noinline__ void set_left_delta(WarpDP &w, int e, int d, int last, int &leftover, int &tEnd, int tLen) {
  const int  lane = threadIdx.x & 31;
  int *const ld   = w.sc.deltaL;
  int n;
  leftover = trace_rows(w, e, d, last, ld, n);
  __syncwarp();
  if (n > 1 && ld[0] == 1 && tEnd + tLen > 0) {
    const int l1 = ld[1];
    __syncwarp();
    for (int i0 = 2; i0 < n; i0 += 32) {   // drop the first entry
      const int i = i0 + lane;
      const int v = i < n ? ld[i] : 0;
      __syncwarp();
      if (i < n) ld[i - 1] = v;
      __syncwarp();
    }
    if (lane == 0) ld[0] = (l1 > 0) ? l1 + 1 : l1 - 1;
    n--;
    tEnd--;
    __syncwarp();
  }
  w.leftLen = n;
}

// Max_Score bookkeeping of forward()/reverse() (prefixEditDistance-forward.C:284-296,
// -reverse.C:300-312), replayed once after the rows instead of on every row.  Row e
// (1..eLast) stored its largest kept value in rowHdr[e].w.  Walking the rows in order,
// the reference scores a row only when that value passes every earlier row's
// (Longest grows) and keeps the first row whose score fl(fl(value * BMV) - e) is the
// strict maximum above the initial 0.0.  Here lane i takes rows i+1, i+33, ...; a warp
// max-scan finds the rows where Longest grows, each lane scores its rows in IEEE double
// (the same two roundings), and a warp arg-max with the smallest row on ties picks the
// reference's row.  msD is the first diagonal of that row's kept band holding msLen.
static __device__ __noinline__ void max_score_rows(const WarpDP &w, int eLast, double &maxScore, int &msLen,
                                                   int &msD, int &msE) {
  const int    lane = threadIdx.x & 31;
  const double BMV  = w.P.branchMatchValue;
  double best  = 0.0;
  int    bestE = INT_MAX;
  int    carry = 0;   // Longest before the current block of 32 rows
  for (int base = 1; base <= eLast; base += 32) {
    const int e = base + lane;
    const int v = e <= eLast ? w.sc.rowHdr[e].w : INT_MIN;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl = max(incl, t);
    }
    int excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = INT_MIN;
    if (e <= eLast && v > max(carry, excl)) {
      const double s = __dsub_rn(__dmul_rn((double)v, BMV), (double)e);
      if (s > best) {
        best  = s;
        bestE = e;
      }
    }
    carry = max(carry, __shfl_sync(0xffffffffu, incl, 31));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int    oe = __shfl_xor_sync(0xffffffffu, bestE, o);
    if (ob > best || (ob == best && oe < bestE)) {
      best  = ob;
      bestE = oe;
    }
  }
  if (bestE == INT_MAX) {
    maxScore = 0.0;
    msLen = msD = msE = 0;
    return;
  }
  maxScore     = best;
  msE          = bestE;
  const int4 h = w.sc.rowHdr[msE];
  msLen        = h.w;
  int myD = INT_MAX;
  for (int d = h.y + lane; d <= h.z; d += 32)
    if (w.sc.arena[h.x + d - h.y] == msLen) {
      myD = d;
      break;
    }
  msD = __reduce_min_sync(0xffffffffu, myD);
}

// ---------------------------------------------------------------------------------
// Row loop of forward()/reverse() (prefixEditDistance-forward.C:131-304,
// -reverse.C:151-320): error rows e = 1, 2, ... with the band pruned against
// Edit_Match_Limit.  It stops at the first row where a diagonal reaches the end of A
// or T (kRowsEnd), when every diagonal is pruned or the error limit is reached
// (kRowsDone), or on a capacity limit (kRowsErr).  Every kept row goes to the arena
// with its largest value in the row header (see max_score_rows).
enum { kRowsDone = 0, kRowsEnd = 1, kRowsErr = 2 };

struct RowsOut {
  int  status;
  u32  err;
  int  e, dEnd, eDone;       // end row, first diagonal reaching an end, last kept row
  int  Rc;                   // right edge of the end row's computed band
  int  rowEnd, ppEnd;        // value of the end row at dEnd, of the row before it at dEnd + 1
  unsigned long long cells, rows;
};

// Several warps of one CTA on one pair (the wide bins): warp 0 runs the pair logic and
// hands each extension's row loop to the whole CTA through GroupShared.
struct GroupJob {
  SeqView    A, T;
  int        a0, t0;
  int        m, n, errorLimit, u;
  int       *rowA, *rowB;    // row buffers (rowA holds row 0), bufW ints each
  int       *rowsG;          // HBM row buffers, rowsGW ints each
  int       *arena;
  int4      *rowHdr;
  const int *eml;
  int        bufW, rowsGW, arenaCap, rowCap;
};
struct GroupShared {
  __align__(16) int  red[2][32][4];   // per-warp partial reductions of a row, by its parity
  GroupJob           job;
  RowsOut            out;             // the row loop's result
  unsigned long long slides;          // slide bases of the CTA's row loops
  int                cmd;             // kGroupRows or kGroupExit, posted by warp 0 before barrier 1
};
enum { kGroupRows = 1, kGroupExit = 2 };

// Named barrier over the CTA's nThr threads (id 1: hand-off, id 2: rows).
__device__ __forceinline__ void group_bar(int id, int nThr) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(nThr) : "memory");
}

// Shared memory of a warp's row loop, in ints: two rows of kRowW diagonals, each with
// kRowPad ints behind it, and the RowJob.
constexpr int kRowW      = 512;
constexpr int kRowPad    = 8;
constexpr int kRowStride = kRowW + kRowPad;

// A row loop's arguments, state between calls and results, in shared memory: what it needs
// rarely or only for addresses stays out of its registers.
struct RowJob {
  SeqView    A, T;
  int       *arena;
  int4      *rowHdr;
  const int *eml;
  int        a0, t0;
  int        arenaCap, bufW;
  int        e, L, R, off, base;   // the row to compute; kept band, place and buffer origin of the row before it
  int        dEnd, Rc, rowEnd, ppEnd;
  u32        cells;
  u32        slides[32];           // per lane
};
constexpr int kJobInts      = (sizeof(RowJob) + 15) / 16 * 4;
constexpr int kWarpSmemInts = 2 * kRowStride + kJobInts;
static_assert(2 * kRowStride % 4 == 0, "RowJob starts on 16 bytes");

// match_run32 of the job's sequences, their planes in registers.
template <bool HASN>
__device__ __forceinline__ int match_len(const RowJob &job, const uint2 *Ap, int ga, const uint2 *Tp, int gt) {
  const uint2 x = load_planes(Ap, ga), y = load_planes(Tp, gt);
  u32 m = (x.x ^ y.x) | (x.y ^ y.y);
  if (HASN) m = drop_n(m, job.A.nm, ga, job.T.nm, gt);
  return __clz((int)m);
}

// Rows e, e + 1, ... by one warp, from the kept band [L, R] of row e - 1 in the buffer
// `prev` (first diagonal `base`, arena place `off`).  Buffers of bufW ints.  Returns a
// RowsOut status, or kRowsWiden when the band outgrew the buffers: row e - 1 is then in the
// buffer of its parity, and the caller continues in wider ones (WIDE: those in HBM).  A row
// buffer holds diagonal d at index d - base + 2, with the two diagonals on each side of the
// kept band set to -2 as the reference does (forward.C:150-153), so the neighbour reads
// need no bounds tests.
//
// What bounds it: instruction issue (63 % of the slots) and the latency of a row.  A row of
// the 2 % reads is 104 diagonals and issues 487 warp instructions, a fifth of them moves of
// the address descriptors that every load of a called function needs.  Measured on the way
// here (DP of 150 Mbp of 0.5 % reads; 20 Mbp of 2 % reads; 4 Mbp of noisy reads):
//   interleaved 2-bit words, the longest slide alone, 32 bases per step, on teams' SMs
//     shared by three CTAs: 648 / 346 / 523 ms;
//   bit planes, long slides by the warp: 426 / 321 / 504 ms; as a team (oic_pairs.cu) and
//     with hopeless groups settled together: 120 / 189 / 127 ms;
//   lanes past the band repeating its last diagonal instead of being masked, one vote for
//     everything rare, the band's edges by two warp reductions per row: 126 / 159 / 54 ms;
//   both directions on forward windows (to the left on the reverse complements), planes
//     with the first base topmost: 107 / 149 / 49 ms.
// A copy of the loop per direction and chunk missed the instruction cache (601 / 377 / 754
// ms before teams).  32 diagonals per step issue as many instructions and wait longer (111 /
// 169 / 56 ms).  Keeping each diagonal's mismatch mask from row to row does not pay: inside
// the band every diagonal moves as fast as the alignment does, so a mask of 32 bases is
// used up in a row or two.
enum { kRowsWiden = 3 };
template <bool HASN, bool WIDE>
static __device__ __noinline__ int row_loop(RowJob &job, const int smOff, int *rowsG, const int m, const int n,
                                            const int errorLimit) {
  const int lane = threadIdx.x & 31;
  int *prev = WIDE ? rowsG : smemRows + smOff, *cur = WIDE ? rowsG + job.bufW : prev + kRowStride;
  const uint2 *const Ap = job.A.p, *const Tp = job.T.p;
  int4 *const rowHdr = job.rowHdr;
  const int *const eml = job.eml;
  const int  a0 = job.a0, t0 = job.t0;
  const int  bufW = job.bufW, arenaCap = job.arenaCap;
  int *const arena = job.arena;
  __builtin_assume(__isGlobal(rowHdr));
  __builtin_assume(__isGlobal(arena));
  __builtin_assume(__isGlobal(eml));
  int e = job.e, L = job.L, R = job.R, off = job.off, base = job.base;
  int lim = e <= errorLimit ? eml[e] : 0;
  u32 cells = 0, slides = 0;
  int status = kRowsDone;
  for (; e <= errorLimit; e++) {
    if (off + R - L + 1 > arenaCap) { status = kRowsErr; break; }
    const int Lc = max(L - 1, -e), Rc = min(R + 1, e);
    const int width = Rc - Lc + 1;
    if (width + 4 > bufW) { status = kRowsWiden; break; }
    const int limNext = e < errorLimit ? eml[e + 1] : 0;
    const int *pv = prev + (2 - base);        // pv[d] = row e-1 at diagonal d
    int       *cv = cur + (2 - Lc);           // cv[d] = row e at diagonal d
    int       *av = arena + (off - L);        // av[d]: row e-1's place in the arena
    int myL = INT_MAX, myR = INT_MIN, prevMax = -1, dEnd = INT_MAX;
#pragma unroll 1
    for (int c = Lc; c <= Rc; c += 64) {
      // Lanes past the band repeat its last diagonal: what they compute and store is what
      // that diagonal's lane computes and stores.
      const int da = min(c + lane, Rc);
      const int pa = pv[da + 1], qa = pv[da];
      int ra = max(max(qa, pa) + 1, pv[da - 1]);
      if (da >= L && da <= R) av[da] = qa;    // keep row e-1 for the traceback
      prevMax = max(prevMax, qa);
      const int za = min(m, n - da);          // where the nearer end is: ra <= za, as no cell of row e-1 is at one
      int sa = ra + match_len<HASN>(job, Ap, a0 + ra, Tp, t0 + da + ra);
      int db = 0, pb = 0, rb = -(1 << 28), zb = INT_MAX, sb = rb;
      if (c + 32 <= Rc) {
        db = min(c + 32 + lane, Rc);
        const int qb = pv[db];
        pb = pv[db + 1];
        rb = max(max(qb, pb) + 1, pv[db - 1]);
        if (db <= R) av[db] = qb;             // db > Lc + 31 >= L
        prevMax = max(prevMax, qb);
        zb = min(m, n - db);
        sb = rb + match_len<HASN>(job, Ap, a0 + rb, Tp, t0 + db + rb);
      }
      if (__any_sync(0xffffffffu, sa >= min(za, ra + 32) || sb >= min(zb, rb + 32))) {
        // A slide through its whole window, or up to an end.
        unsigned moreA = __ballot_sync(0xffffffffu, c + lane <= Rc && sa == ra + 32 && sa < za);
        unsigned moreB = __ballot_sync(0xffffffffu, c + 32 + lane <= Rc && sb == rb + 32 && sb < zb);
        while (moreA | moreB) {
          // One lane's slide goes on: the warp looks at 32 windows of 32 bases per step.
          const bool second = moreA == 0;
          const unsigned w = second ? moreB : moreA;
          const int  q  = __ffs((int)w) - 1;
          const int  zq = __shfl_sync(0xffffffffu, second ? zb : za, q);
          const int  dq = c + q + (second ? 32 : 0);
          if (second) moreB = w & (w - 1);
          else moreA = w & (w - 1);
          for (int r = __shfl_sync(0xffffffffu, second ? sb : sa, q);; r += 1024) {
            const int at = r + 32 * lane;
            int len = 0;
            if (at < zq) len = match_len<HASN>(job, Ap, a0 + at, Tp, t0 + dq + at);
            const unsigned stop = __ballot_sync(0xffffffffu, len < 32);
            if (stop) {
              const int f  = __ffs((int)stop) - 1;
              const int to = __shfl_sync(0xffffffffu, at + len, f);
              if (dq == (second ? db : da)) {   // the lane, and those that repeat it
                if (second) sb = to;
                else sa = to;
              }
              break;
            }
          }
        }
        if (dEnd == INT_MAX) {
          const unsigned endA = __ballot_sync(0xffffffffu, sa >= za), endB = __ballot_sync(0xffffffffu, sb >= zb);
          if (endA | endB) {
            const int f = __ffs((int)(endA ? endA : endB)) - 1;
            dEnd = c + f + (endA ? 0 : 32);
            if (lane == f) {
              job.rowEnd = endA ? za : zb;
              job.ppEnd  = endA ? pa : pb;
            }
          }
        }
      }
      sa = min(sa, za);
      sb = min(sb, zb);
      cv[da] = sa;
      if (c + 32 <= Rc) cv[db] = sb;
      if (c + lane <= Rc) slides += (u32)(sa - ra);
      if (c + 32 + lane <= Rc) slides += (u32)(sb - rb);
      // pruneAlign (prefixEditDistance.H:249-258): extra = max(d, 0) on both band edges
      if (sa + max(da, 0) >= lim) {
        myL = min(myL, da);
        myR = da;
      }
      if (sb + max(db, 0) >= lim) {
        myL = min(myL, db);
        myR = db;
      }
    }
    // Row e-1's header, with its largest value (forward.C:284-289) for max_score_rows.
    prevMax = __reduce_max_sync(0xffffffffu, prevMax);
    if (lane == 0) rowHdr[e - 1] = make_int4(off, L, R, prevMax);
    if (dEnd != INT_MAX) {
      cells += (u32)(dEnd - Lc + 1);
      status = kRowsEnd;
      if (lane == 0) {
        job.dEnd = dEnd;
        job.Rc   = Rc;
      }
      break;
    }
    cells += (u32)width;
    // The kept band is [first, last] unpruned diagonal (forward.C:245-280).
    const int L2 = __reduce_min_sync(0xffffffffu, myL), R2 = __reduce_max_sync(0xffffffffu, myR);
    if (L2 == INT_MAX) break;
    __syncwarp();
    if (lane < 4) cv[lane < 2 ? L2 - 2 + lane : R2 - 1 + lane] = -2;
    off += R - L + 1;
    int *t = prev;
    prev   = cur;
    cur    = t;
    base   = Lc;
    L      = L2;
    R      = R2;
    lim    = limNext;
    __syncwarp();
  }
  if (e > errorLimit) {
    // The error limit: the last row has not been kept yet.
    if (off + R - L + 1 > arenaCap) status = kRowsErr;
    else {
      const int *pv = prev + (2 - base);
      int prevMax = -1;
      for (int d = L + lane; d <= R; d += 32) {
        const int v = pv[d];
        arena[off + d - L] = v;
        prevMax            = max(prevMax, v);
      }
      prevMax = __reduce_max_sync(0xffffffffu, prevMax);
      if (lane == 0) rowHdr[errorLimit] = make_int4(off, L, R, prevMax);
    }
  }
  __syncwarp();
  if (lane == 0) {
    job.e    = e;
    job.L    = L;
    job.R    = R;
    job.off  = off;
    job.base = base;
    job.cells += cells;
  }
  job.slides[lane] += slides;
  __syncwarp();
  return status;
}

// The row loop by one warp: rows in shared memory, and in the warp's HBM rows from the row
// on whose band has outgrown them.  r0: row 0's value.
static __device__ __noinline__ void warp_rows(WarpDP &w, RowsOut &o, const SeqView &A, int a0, int m, const SeqView &T,
                                              int t0, int n, int errorLimit, int r0) {
  const int  lane = threadIdx.x & 31;
  int *const bufA = smemRows + w.smOff, *const bufB = bufA + kRowStride;
  RowJob    &job  = *(RowJob *)(bufB + kRowStride);
  const int  rowCap = w.cap.rowCap, gw = w.cap.rowsGW;
  int *const rowsG  = w.sc.rowsG;
  const bool hasN   = A.nm || T.nm;
  if (lane < 5) bufA[lane] = lane == 2 ? r0 : -2;
  if (lane == 0) {
    job.A        = A;
    job.T        = T;
    job.arena    = w.sc.arena;
    job.rowHdr   = w.sc.rowHdr;
    job.eml      = w.eml;
    job.a0       = a0;
    job.t0       = t0;
    job.arenaCap = w.cap.arenaCap;
    job.bufW     = kRowW;
    job.e        = 1;
    job.L = job.R = job.off = job.base = 0;
    job.cells    = 0;
  }
  job.slides[lane] = 0;
  __syncwarp();
  // Row rowCap has no header: the loop stops before it.
  const bool capped = errorLimit >= rowCap;
  const int  limit  = capped ? rowCap - 1 : errorLimit;
  u32 err = kErrArenaFull;
  int st  = hasN ? row_loop<true, false>(job, w.smOff, rowsG, m, n, limit)
                 : row_loop<false, false>(job, w.smOff, rowsG, m, n, limit);
  if (st == kRowsWiden) {
    if (job.R - job.L + 7 > gw || !rowsG) {
      st  = kRowsErr;
      err = kErrBandWide;
    } else {
      const int *src = (job.e & 1) ? bufA : bufB;   // even rows are in bufA
      for (int i = lane; i < kRowW; i += 32) rowsG[i] = src[i];
      if (lane == 0) job.bufW = gw;
      __syncwarp();
      st = hasN ? row_loop<true, true>(job, w.smOff, rowsG, m, n, limit)
                : row_loop<false, true>(job, w.smOff, rowsG, m, n, limit);
      if (st == kRowsWiden) {
        st  = kRowsErr;
        err = kErrBandWide;
      }
    }
  }
  const int e = job.e;
  if (capped && e > limit && st == kRowsDone) {
    st  = kRowsErr;
    err = kErrRowsFull;
  }
  o.status = st;
  o.err    = st == kRowsErr ? err : 0;
  o.e      = e;
  o.eDone  = e - 1;      // rows below e are kept
  o.dEnd   = job.dEnd;
  o.Rc     = job.Rc;
  o.rowEnd = job.rowEnd;
  o.ppEnd  = job.ppEnd;
  o.cells  = job.cells;
  o.rows   = (unsigned)(e <= limit && st != kRowsErr ? e : e - 1);   // row e itself was computed when the loop ended in it
  w.slides += job.slides[lane];
  __syncwarp();
}

// ---------------------------------------------------------------------------------
// True when no alignment of S and T with at most E errors runs from the start of S or T to
// the end of S or T and, on the way, through a point on a diagonal (T offset - S offset) of
// [dlo, dhi] that it reaches within those errors: then no match node on those diagonals
// whose error limit is at most E extends to both ends.  (False says nothing.)
//
// One wavefront over all of them: row e holds, for each diagonal, the furthest S position
// that e errors reach from any start on the boundary.  Every alignment of the statement is
// followed: with e errors used it is at most E - e diagonals beside [dlo, dhi] if the point
// is still ahead, and at most e if it lies behind, so row e needs only the diagonals within
// max(E - e, e).  Nothing else is pruned, so reaching an end row is the only way out.  Cells
// that no alignment has reached hold a large negative value.
//
// The row is updated in place in the warp's row buffers (nDiag <= kProofDiags), 64 diagonals
// per step: a step's loads, the old value to its left among them, come before its stores.
constexpr int kProofDiags = 2 * kRowStride - 4;
static __device__ __noinline__ bool no_path_within(WarpDP &w, const ReadView &Sref, int sLen, const ReadView &Tref,
                                                   int tLen, int dlo, int dhi, int E) {
  const SeqView S = Sref.f, T = Tref.f;
  const int lane  = threadIdx.x & 31;
  constexpr int kFar = -(1 << 28);
  const int lo = max(dlo - E, 1 - sLen), hi = min(dhi + E, tLen - 1);
  int *const v = smemRows + w.smOff + 1 - lo;   // v[d], d in [lo - 1, hi + 1]
  for (int d = lo - 1 + lane; d <= hi + 1; d += 32) v[d] = kFar;
  __syncwarp();
  u32 cells = 0;
  bool end  = false;
  int  e    = 0;
  for (; e <= E && !end; e++) {
    const int W  = max(E - e, e);
    const int dL = max(lo, dlo - W), dR = min(hi, dhi + W);
    int left = v[dL - 1];                       // old value left of the step
#pragma unroll 1
    for (int c = dL; c <= dR; c += 64) {
      const int  da = min(c + lane, dR), db = min(c + 32 + lane, dR);
      const bool ina = c + lane <= dR, inb = c + 32 + lane <= dR;
      const int  a0 = v[da], a1 = v[da + 1], b0 = v[db], b1 = v[db + 1];
      int am = __shfl_up_sync(0xffffffffu, a0, 1), bm = __shfl_up_sync(0xffffffffu, b0, 1);
      const int a31 = __shfl_sync(0xffffffffu, a0, 31);
      if (lane == 0) {
        am = left;
        bm = a31;
      }
      left = __shfl_sync(0xffffffffu, b0, 31);
      int ra = e ? max(max(a0, a1) + 1, am) : max(0, -da);
      int rb = e ? max(max(b0, b1) + 1, bm) : max(0, -db);
      const bool oka = ina && ra >= 0, okb = inb && rb >= 0;
      const int  ka = min(sLen - ra, tLen - da - ra), kb = min(sLen - rb, tLen - db - rb);
      int sa = 0, sb = 0;
      if (oka) sa = match_run32(S, ra, T, ra + da);
      if (okb) sb = match_run32(S, rb, T, rb + db);
      // Slides past a window go on 32 bases per step (the first half's, then the second's).
      bool fa = oka && sa == 32 && ka > 32, fb = okb && sb == 32 && kb > 32;
      while (__any_sync(0xffffffffu, fa || fb)) {
        if (fa || fb) {
          const int r   = fa ? ra + sa : rb + sb;
          const int len = match_run32(S, r, T, r + (fa ? da : db));
          if (fa) {
            sa += len;
            fa = len == 32 && sa < ka;
          } else {
            sb += len;
            fb = len == 32 && sb < kb;
          }
        }
      }
      __syncwarp();
      if (ina) v[da] = oka ? ra + min(sa, ka) : kFar;
      if (inb) v[db] = okb ? rb + min(sb, kb) : kFar;
      end |= __any_sync(0xffffffffu, (oka && sa >= ka) || (okb && sb >= kb));
    }
    cells += (u32)(dR - dL + 1);
    __syncwarp();
    // The cells beside the row are not part of it (they hold row e - 1's edge cells).
    if (lane == 0) {
      v[dL - 1] = kFar;
      v[dR + 1] = kFar;
    }
    __syncwarp();
  }
  w.cells += cells;
  w.rows += (u32)e;
  return !end;
}

// The row loop by every thread of the CTA (nThr threads, tid = threadIdx.x).  Thread t
// takes diagonals Lc + t, Lc + t + nThr, ..., U of them per pass, their loads together.
// Every decision is made on CTA-reduced values, so all threads take the same path and
// meet the same barriers.
//
// What bounds it is the latency of a row: shared-memory loads, the windows, a barrier and
// the reduction behind it.  One barrier per row: the partial reductions go to slots of the
// row's parity, neighbours outside the kept band are masked instead of overwritten, and the
// kept band goes to the arena (with its largest value to the header) while the next row
// reads it, as in row_loop.  A batch of 230 extensions of 60 kb reads with 4 % errors took
// 39.6 ms with a sentinel write, a copy of the kept band and four barriers per row (and
// one-warp rows in HBM first, for bands that end up here), 26.3 ms with one barrier, 19.4 ms
// with the job read from shared memory, 14.2 ms with 512 threads instead of 256.  Two CTAs
// of 512 threads per SM (64 registers) spill: 18.0 ms.
template <int U, bool HASN>
static __device__ __noinline__ void group_rows(GroupShared &gs, const int tid, const int nThr) {
  const int lane = tid & 31, wid = tid >> 5;
  const GroupJob &j = gs.job;
  // The planes in registers for the slides (N masks are read from the job when needed).
  const uint2 *const Ap = j.A.p + 0, *const Tp = j.T.p + 0;
  const int a0 = j.a0, t0 = j.t0, m = j.m, n = j.n, errorLimit = j.errorLimit;
  const int arenaCap = j.arenaCap, rowCap = j.rowCap;
  int4 *const rowHdr = j.rowHdr;
  int  *const arena  = j.arena;
  const int *const eml = j.eml;
  __builtin_assume(__isGlobal(rowHdr));
  __builtin_assume(__isGlobal(arena));
  __builtin_assume(__isGlobal(eml));
  int *prev = j.rowA, *cur = j.rowB;   // diagonal d at index d - base + 2
  int  bufW = j.bufW;
  int  off = 0, base = 0, L = 0, R = 0;
  int  lim = errorLimit >= 1 ? eml[1] : 0;
  int  e = 1, status = kRowsDone;
  u32  err = 0, cells = 0, slides = 0;
  for (; e <= errorLimit; e++) {
    if (e >= rowCap) { status = kRowsErr; err = kErrRowsFull; break; }
    if (off + (R - L + 1) > arenaCap) { status = kRowsErr; err = kErrArenaFull; break; }
    const int Lc = max(L - 1, -e), Rc = min(R + 1, e);
    const int width = Rc - Lc + 1;
    if (width + 4 > bufW) {
      int *const rowsG = j.rowsG;
      const int  gw    = j.rowsGW;
      if (bufW == gw || width + 4 > gw || !rowsG) { status = kRowsErr; err = kErrBandWide; break; }
      for (int i = tid; i < bufW; i += nThr) rowsG[i] = prev[i];
      group_bar(2, nThr);
      prev = rowsG;
      cur  = rowsG + gw;
      bufW = gw;
    }
    const int limNext = e < errorLimit ? eml[e + 1] : 0;
    int myEnd = INT_MAX, myL = INT_MAX, myR = INT_MIN, prevMax = -1;
    for (int c = Lc + tid; c <= Rc; c += nThr * U) {
      int row[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int d = c + k * nThr;
        if (d <= Rc) {
          // Row e-1 at d - 1, d, d + 1; -2 outside its kept band (forward.C:150-153).
          const int *pv = prev + (2 - base) + d;
          const int  pm = d > L ? pv[-1] : -2, p0 = d >= L && d <= R ? pv[0] : -2, pp = d < R ? pv[1] : -2;
          if (d >= L && d <= R) arena[off - L + d] = p0;
          prevMax = max(prevMax, p0);
          row[k]  = max(max(p0, pp) + 1, pm);
        }
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int d = c + k * nThr;
        if (d <= Rc) {
          const int z = min(m, n - d);   // where the nearer end is
          int r = row[k];
          while (r < z) {
            const uint2 x = load_planes(Ap, a0 + r), y = load_planes(Tp, t0 + d + r);
            u32 mk = (x.x ^ y.x) | (x.y ^ y.y);
            if (HASN) mk = drop_n(mk, j.A.nm, a0 + r, j.T.nm, t0 + d + r);
            r += __clz((int)mk);
            if (mk) break;
          }
          r = min(r, z);
          slides += (u32)(r - row[k]);
          cur[2 - Lc + d] = r;
          if (r == z) myEnd = min(myEnd, d);
          // pruneAlign (prefixEditDistance.H:249-258): extra = max(d, 0) on both band edges
          if (r + max(d, 0) >= lim) {
            myL = min(myL, d);
            myR = d;
          }
        }
      }
    }
    int (*const slot)[4] = gs.red[e & 1];
    {
      const int wEnd = __reduce_min_sync(0xffffffffu, myEnd);
      const int wL   = __reduce_min_sync(0xffffffffu, myL);
      const int wR   = __reduce_max_sync(0xffffffffu, myR);
      const int wV   = __reduce_max_sync(0xffffffffu, prevMax);
      if (lane == 0) *(int4 *)slot[wid] = make_int4(wEnd, wL, wR, wV);
    }
    group_bar(2, nThr);
    // Every warp reduces the warps' results: lane i takes warp i's.
    int4 w = make_int4(INT_MAX, INT_MAX, INT_MIN, -1);
    if (lane < nThr >> 5) w = *(const int4 *)slot[lane];
    const int dEnd = __reduce_min_sync(0xffffffffu, w.x);
    const int L2   = __reduce_min_sync(0xffffffffu, w.y);
    const int R2   = __reduce_max_sync(0xffffffffu, w.z);
    prevMax        = __reduce_max_sync(0xffffffffu, w.w);
    // Row e-1's header, with its largest value (forward.C:284-289) for max_score_rows.
    if (tid == 0) rowHdr[e - 1] = make_int4(off, L, R, prevMax);
    if (dEnd != INT_MAX) {
      cells += (u32)(dEnd - Lc + 1);
      status = kRowsEnd;
      if (tid == 0) {
        gs.out.dEnd   = dEnd;
        gs.out.Rc     = Rc;
        gs.out.rowEnd = cur[2 - Lc + dEnd];
        gs.out.ppEnd  = dEnd < R ? prev[2 - base + dEnd + 1] : -2;
      }
      break;
    }
    cells += (u32)width;
    if (L2 == INT_MAX) break;
    off += R - L + 1;
    int *t = prev;
    prev   = cur;
    cur    = t;
    base   = Lc;
    L      = L2;
    R      = R2;
    lim    = limNext;
  }
  if (e > errorLimit) {
    // The error limit: the last row has not been kept yet.
    if (off + (R - L + 1) > arenaCap) {
      status = kRowsErr;
      err    = kErrArenaFull;
    } else {
      int prevMax = -1;
      for (int d = L + tid; d <= R; d += nThr) {
        const int v = prev[2 - base + d];
        arena[off + d - L] = v;
        prevMax            = max(prevMax, v);
      }
      prevMax = __reduce_max_sync(0xffffffffu, prevMax);
      if (lane == 0) gs.red[e & 1][wid][3] = prevMax;
      group_bar(2, nThr);
      for (int i = 0; i < nThr >> 5; i++) prevMax = max(prevMax, gs.red[e & 1][i][3]);
      if (tid == 0) rowHdr[errorLimit] = make_int4(off, L, R, prevMax);
    }
  }
  const unsigned long long sl = warp_sum64(slides);
  if (lane == 0) atomicAdd(&gs.slides, sl);
  if (tid == 0) {
    gs.out.status = status;
    gs.out.err    = err;
    gs.out.e      = e;
    gs.out.eDone  = e - 1;   // rows below e are kept
    gs.out.cells  = cells;
    gs.out.rows   = (unsigned)(e <= errorLimit && status != kRowsErr ? e : e - 1);
  }
  // Warp 0 goes on alone with the arena and the buffers: everything has been written.
  __threadfence_block();
  group_bar(2, nThr);
}

// The posted job, with its compile-time tile.
static __device__ __forceinline__ void group_rows_any(GroupShared &gs, int tid, int nThr) {
  const bool hasN = gs.job.A.nm || gs.job.T.nm;
  const int  u    = gs.job.u;
  if (hasN) group_rows<1, true>(gs, tid, nThr);
  else if (u == 4) group_rows<4, false>(gs, tid, nThr);
  else if (u == 2) group_rows<2, false>(gs, tid, nThr);
  else group_rows<1, false>(gs, tid, nThr);
}

// Worker warps of a group CTA: run the row loops warp 0 posts until it posts exit.
static __device__ __noinline__ void group_worker(GroupShared &gs) {
  while (true) {
    group_bar(1, blockDim.x);
    if (gs.cmd != kGroupRows) break;
    group_rows_any(gs, threadIdx.x, blockDim.x);
  }
}

// forward() (prefixEditDistance-forward.C:94-314) for step = +1 and reverse()
// (prefixEditDistance-reverse.C:114-330) for step = -1.  A[i] is base a0+i of view A,
// T likewise (for step = -1 the reads' reverse complements).  The row loop runs on this warp, or on the whole CTA when w.gs is
// set (warp 0 of a group CTA); the rest runs on this warp.  Returns the error count;
// the outputs are warp-uniform.  On a capacity overflow sets w.err and returns 0.
// endOnly: the caller uses the outputs only when the end is reached (toEnd); otherwise
// they are not computed.
template <bool GROUP>
static __device__ __noinline__ int warp_prefix_dp(WarpDP &w, const int step, const SeqView &A, int a0, int m, const SeqView &T, int t0, int n,
                              int errorLimit, bool endOnly, int &aEnd, int &tEnd, int &leftover, bool &toEnd) {
  const int lane = threadIdx.x & 31;
  const double BMV = w.P.branchMatchValue;

  if (step > 0) w.rightLen = 0;
  else w.leftLen = 0;

  const int r0 = warp_slide0(A, a0, T, t0, m, w.slides);
  if (r0 == m) {
    aEnd = tEnd = step * m;
    if (step < 0) leftover = m;
    toEnd = true;
    return 0;
  }

  RowsOut o;
  if (GROUP) {
    if (lane == 0) {
      w.smA[2]     = r0;
      GroupJob &j  = w.gs->job;
      j.A          = A;
      j.T          = T;
      j.a0         = a0;
      j.t0         = t0;
      j.m          = m;
      j.n          = n;
      j.errorLimit = errorLimit;
      j.u          = w.gU;
      j.rowA       = w.smA;
      j.rowB       = w.smB;
      j.rowsG      = w.sc.rowsG;
      j.arena      = w.sc.arena;
      j.rowHdr     = w.sc.rowHdr;
      j.eml        = w.eml;
      j.bufW       = w.cap.bandW;
      j.rowsGW     = w.cap.rowsGW;
      j.arenaCap   = w.cap.arenaCap;
      j.rowCap     = w.cap.rowCap;
      w.gs->cmd    = kGroupRows;
    }
    __syncwarp();
    group_bar(1, w.gThreads);
    group_rows_any(*w.gs, lane, w.gThreads);
    o = w.gs->out;
  } else {
    warp_rows(w, o, A, a0, m, T, t0, n, errorLimit, r0);
  }
  w.cells += o.cells;
  w.rows += o.rows;
  if (o.status == kRowsErr) {
    w.err |= o.err;
    return 0;
  }
  if (endOnly && o.status != kRowsEnd) {
    toEnd = false;
    return 0;
  }

  double maxScore = 0.0;
  int    msLen = 0, msD = 0, msE = 0;
  max_score_rows(w, o.eDone, maxScore, msLen, msD, msE);

  if (o.status == kRowsEnd) {
    const int e   = o.e;
    const int row = o.rowEnd;
    // Branch-point test in IEEE double on lane 0 (the FP64 pipe is narrow); the other
    // lanes take its decision.
    int abort_ = 0;
    if (lane == 0) {
      const double score   = __dsub_rn(__dmul_rn((double)row, BMV), (double)e);
      const int    tailLen = row - msLen;
      const double slope   = __ddiv_rn(__dsub_rn(maxScore, score), (double)tailLen);
      abort_ = (w.P.partial && score < maxScore) ||
               (e > 20 / 2 && tailLen >= 20 && slope >= w.P.minBranchTailSlope);
    }
    abort_ = __shfl_sync(0xffffffffu, abort_, 0);
    if (!abort_) {
      int d = o.dEnd;
      if (step > 0) {
        // Force the last error to be a mismatch (forward.C:215-221).
        if (row == m && 1 + o.ppEnd == row && d < o.Rc) d++;
        aEnd = row;
        tEnd = row + d;
        set_right_delta(w, e, d, row);
      } else {
        aEnd = -row;
        tEnd = -row - d;
        set_left_delta(w, e, d, row, leftover, tEnd, n);
      }
      toEnd = true;
      return e;
    }
    if (endOnly) {
      toEnd = false;
      return 0;
    }
  }

  // Branch point, errors exhausted, or every diagonal pruned (forward.C:197-212,
  // 306-313): the alignment ends at the Max_Score row.
  aEnd = step * msLen;
  tEnd = step * (msLen + msD);
  const int last = arena_get(w, msE, msD);
  if (step > 0) set_right_delta(w, msE, msD, last);
  else set_left_delta(w, msE, msD, last, leftover, tEnd, n);
  toEnd = false;
  return msE;
}

static __device__ __forceinline__ void warp_dp_init(WarpDP &w, const WarpScratch &sc, const AlignCaps &cap, int smOff,
                                                    const int *eml, const DevParams &P) {
  w.sc       = sc;
  w.cap      = cap;
  w.smOff    = smOff;
  w.smA      = smemRows + smOff;             // a group CTA's two rows of cap.bandW
  w.smB      = w.smA + cap.bandW;
  w.eml      = eml;
  w.P        = P;
  w.cells    = 0;
  w.slides   = 0;
  w.rows     = 0;
  w.err      = 0;
  w.leftLen  = w.rightLen = 0;
  w.gs       = nullptr;
  w.gThreads = 32;
  w.gU       = 1;
}

enum { kNone = 0, kLeftBranch = 1, kRightBranch = 2, kDovetail = 3 };

// Extend_Alignment (prefixEditDistance-extend.C:36-183), one warp.  The merged delta
// ends up in sc.deltaL[0 .. leftLen).  Outputs are warp-uniform.
// dovetailOnly: the caller uses the outputs only when both ends are reached.  The left
// side is then not extended after the right side has failed, and a side that fails is not
// traced: pairs that share only a repeat fail on one side in nearly every extension, and
// on repeat-rich low-error reads they are nine tenths of the cells.
template <bool GROUP>
static __device__ __noinline__ int warp_extend(WarpDP &w, bool dovetailOnly, const ReadView &S, int sLen, const ReadView &T, int tLen, int mStart,
                           int mOffset, int mLen, int &sLo, int &sHi, int &tLo, int &tHi, int &errors) {
  const int lane = threadIdx.x & 31;
  int  rightErrors = 0, leftErrors = 0, leftover = 0;
  bool rToEnd = true, lToEnd = true;
  const int sLeftBegin = mStart - 1, sRightBegin = mStart + mLen, sRightLen = sLen - sRightBegin;
  const int tLeftBegin = mOffset - 1, tRightBegin = mOffset + mLen, tRightLen = tLen - tRightBegin;
  int totalOlap = min(mStart, mOffset) + mLen + min(sRightLen, tRightLen);
  if (totalOlap < 0) totalOlap = 0;
  if (totalOlap > (int)kMaxReadLen) totalOlap = (int)kMaxReadLen;
  const int errorLimit = error_bound(totalOlap, w.P.maxErate);

  w.leftLen = w.rightLen = 0;

  if (sRightLen == 0 || tRightLen == 0) {
    sHi = tHi = 0;
    rToEnd    = true;
  } else if (sRightLen <= tRightLen) {
    rightErrors = warp_prefix_dp<GROUP>(w, +1, S.f, sRightBegin, sRightLen, T.f, tRightBegin, tRightLen, errorLimit,
                                     dovetailOnly, sHi, tHi, leftover, rToEnd);
    if (w.err) return kNone;
    for (int i = lane; i < w.rightLen; i += 32) w.sc.deltaR[i] = -w.sc.deltaR[i];
  } else {
    rightErrors = warp_prefix_dp<GROUP>(w, +1, T.f, tRightBegin, tRightLen, S.f, sRightBegin, sRightLen, errorLimit,
                                     dovetailOnly, tHi, sHi, leftover, rToEnd);
    if (w.err) return kNone;
  }
  if (dovetailOnly && !rToEnd) return kNone;
  __syncwarp();
  sHi += sRightBegin - 1;
  tHi += tRightBegin - 1;

  leftover = 0;
  if (sLeftBegin < 0 || tLeftBegin < 0) {
    sLo = tLo = 0;
    lToEnd    = true;
  } else if (sRightBegin <= tRightBegin) {
    leftErrors = warp_prefix_dp<GROUP>(w, -1, S.c, sLen - mStart, sLeftBegin + 1, T.c, tLen - mOffset, tLeftBegin + 1,
                                    errorLimit - rightErrors, dovetailOnly, sLo, tLo, leftover, lToEnd);
    if (w.err) return kNone;
  } else {
    leftErrors = warp_prefix_dp<GROUP>(w, -1, T.c, tLen - mOffset, tLeftBegin + 1, S.c, sLen - mStart, sLeftBegin + 1,
                                    errorLimit - rightErrors, dovetailOnly, tLo, sLo, leftover, lToEnd);
    if (w.err) return kNone;
    for (int i = lane; i < w.leftLen; i += 32) w.sc.deltaL[i] = -w.sc.deltaL[i];
  }
  if (dovetailOnly && !lToEnd) return kNone;
  __syncwarp();
  sLo += sLeftBegin + 1;
  tLo += tLeftBegin + 1;
  errors = leftErrors + rightErrors;

  const int kind = (!rToEnd) ? ((!lToEnd) ? kNone : kRightBranch) : ((!lToEnd) ? kLeftBranch : kDovetail);

  // Merge the right delta into the left one (extend.C:164-175).
  if (w.leftLen + w.rightLen + 1 > w.cap.rowCap) { w.err |= kErrDeltaFull; return kNone; }
  if (w.rightLen > 0) {
    const int base = w.leftLen;
    if (lane == 0) {
      const int r0 = w.sc.deltaR[0];
      w.sc.deltaL[base] = (r0 > 0) ? -(r0 + leftover + mLen) : -(r0 - leftover - mLen);
    }
    for (int i = 1 + lane; i < w.rightLen; i += 32) w.sc.deltaL[base + i] = -w.sc.deltaR[i];
    w.leftLen = base + w.rightLen;
  }
  w.rightLen = 0;
  __syncwarp();
  return kind;
}

}  // namespace oic

// dc_recolor.cu -- seeding + recolouring loop of one update batch, as one
// cooperative persistent launch with software grid barriers.
//
// Snapshot schedule: every reference kernel launch is one step whose reads
// see the state at the start of the step.  A step that computes colours
// (REDUCE) writes them to ncolor[]; the following COMMIT step publishes them.
//
//   HI  (HI/gpuFunctions_undir.cuh:147-284, HI/Color_main.cu:146-202)
//     D1  deletions: target = endpoint with the larger colour (tie: node2)
//     D2  mex of every target                           -> ncolor
//     D3  commit where the colour changed; frontier F0 += target
//     I1  insertions whose colours were equal before the batch and still are
//     I2  saturation size (distinct neighbour colours) of both endpoints
//     I3  target = endpoint with the smaller saturation (tie: node2)
//     I4  mex of every target                           -> ncolor
//     I5  commit unconditionally; F0 += target
//   HB  (HB/gpuFunctions_undir.cuh:104-314, HB/Color_main.cu:160-224)
//     H1  every endpoint of (equal-colour insertions + deletions)
//     H2  mex over neighbours prior in LDF order        -> ncolor
//     H3  commit where the colour changed; F0 += vertex
//   loop (both), until the frontier is empty (HI) or nothing changed (HB).
//   The reference's step is findEligibleNeighbors over the frontier F (marks
//   the next frontier Q), recolorNeighbor over Q, commit, F = Q.  Q is found
//   without walking every row of F, and a mex is computed only where it can
//   have changed; both give exactly the reference's sets and colours:
//     MARK    PUSH: rows of the frontier vertices that are new, or (HI) whose
//             colour or previous colour changed, mark their neighbours; rows
//             whose colour changed make the neighbours it matters to dirty.
//             PULL, beside it: every member u of F keeps its place in Q when
//             its witness (a neighbour that marked it before) still does, or
//             another neighbour does; otherwise it leaves
//     EVAL    mex of the dirty vertices of Q -> ncolor.  SCAN, beside it:
//             long rows looking for a new witness, split over many warps
//     COMMIT  colours, frontier flags, the next iteration's PUSH rows
//     APPEND  (HI with the heavy-row index) vertices whose colour changed
//             for the first time join the change lists of their indexed
//             neighbours
//   Why PUSH and PULL find all of Q: a vertex outside F was marked by no
//   frontier vertex in the last step, so only a frontier vertex that is new
//   or whose (colour, previous colour) pair differs from the last step can
//   mark it now; a vertex inside F is tested against all its neighbours.
//   Why a clean mex can be kept: a vertex whose colour is the mex of its
//   (HB: prior) neighbours gets another one only if a neighbour left a
//   smaller colour or took its own.
//   Counted on the oracle's schedule (R-MAT scale 17, 8,192 lines): HI visits
//   16 M adjacency entries where walking the frontier's rows (indexed ones by
//   their candidates) visits 50 M, HB 0.1 G where that visits 0.5 G.  Measured
//   with all of it, ms of device time per batch, before -> after: R-MAT scale
//   24, 1 M lines, HI 157 -> 75; scale 22, 250 k lines, HB 331 -> 69; Chung-Lu
//   1 M vertices, 250 k lines, HB 66 -> 15, HI 17 -> 14; R-MAT scale 16, 20 k
//   lines, HI 4.8 -> 2.9, HB 6.6 -> 3.0.  What bounds the loop then is the
//   chain of dependent L2 round trips in each of its three phases and their
//   barriers, 3.5 us for a phase with nothing to do and 6 to 10 for one with a
//   few rows; and for HB on large graphs the dirty walks (see push_dirty).
//
// Heavy-row index (built by dc_hri.cu before the launch, for batches large
// enough to use it): HI reads an indexed row through its colour-ordered copy
// and change list instead of gathering every neighbour's colour; HB reads
// the prior part of an indexed row where its rule concerns prior neighbours
// and the rest where it concerns the others.
//
// Work is split by row length: rows of <= kSmall slots ("class A") are
// processed 32 at a time by one warp with a warp-level load-balanced search
// over their slots; longer rows become units of up to unit_slots slots, one
// warp per unit.  A row of several units combines its partial colour masks
// in a global mask slot; the unit that finishes last computes the result.
#include "dc_device.cuh"

namespace dc {

namespace {

enum Mode { M_MEX_ALL = 0, M_MEX_PRIOR = 1, M_DISTINCT = 2 };

constexpr int kCtaBuf = 4096, kMemBuf = 1024;  // vertices a CTA stages for a queue and for the member list in a phase

// What the device functions of a launch share, in the CTA's shared memory.
// The code is kept small on purpose: the phases alternate every few
// microseconds, and a kernel with every helper inlined (528 KB of code at
// the start) refetches its instructions from L2 in each of them.  So the
// helpers are calls, and their common arguments live here.
struct Env {
  GraphDev g;
  DevState* st;
  LoopState* ls;     // the loop's counters
  unsigned nwarps;   // warps of the grid
  int loop_units;    // slots per work unit of the loop's rows
  QueueBufs qb[3];
  unsigned* bmA;
  int* ncolor;
  // HB: (degree property << 32) | colour word per vertex, so one 8-byte
  // gather gives both; the frontier flags live in its colour half
  unsigned long long* cp;
  // HB, with the index: each vertex's colour, those of kC8Top or more as
  // kC8Top, for the walks of indexed rows, which need nothing else
  unsigned char* c8;
  HriBufs hri;       // heavy-row index
  bool hri_on;       // HI: index in use
  bool hri_split;    // HB: indexed rows list their prior neighbours first
  // loop
  int* mem;          // frontier member list
  long long mem_cap;
  int* mout;         // members that leave
  int* wit;          // each member's witness
  unsigned* inF;     // frontier membership bits (bmB)
  unsigned* clean;   // set: the colour is the mex of the neighbours (bmC)
  unsigned* inE;     // in the EVAL queue (bmA)
  // batched mode (all nullptr for one graph)
  const int* gid;
  int* gcount;       // HI: frontier vertices per graph
  int* gchg;         // HB: colour changes per graph, this iteration
  const int* gskip;  // HB: graphs whose last recolour step changed nothing have stopped
  int* gf0;          // frontier F0 vertices per graph
};

// Rows of a warp, for walks that spread the slots of up to 32 rows over the
// lanes: where each starts in the slots' numbering and in memory, and what the
// walk needs to know of it.
struct Rows {
  int excl[32];
  const int* at[32];
  int a[32], b[32], c[32], d[32];
};

// Where a launch is in its sequence of phases.
struct Step {
  int ph;         // the phase
  int ps;         // phase count mod 3, for the ring of work counters
  int r, rn;      // it % 3, (it + 1) % 3
  long long it;   // the loop's iteration
};

// The work items of a MARK or EVAL phase: units in 2^us pieces, then (MARK)
// shares of 2^ms members, then class-A batches of 2^as rows.
struct Work {
  unsigned units, members, total;  // items of the first kind, of the first two, of all
  int us, ms, as;
  int sh;                          // log2 of the items a warp takes at a time
};

struct Shared {
  Env E;
  LoopState snap;                     // the loop's counters at the last grid barrier
  unsigned mask[kWarps][kMaskWords];  // per-warp colour window
  Rows rows[kWarps];                  // the rows a warp walks together
  long long scanned[kWarps];          // seeding: live entries the scanned rows cover
  long long idx_cov[kWarps];          // of those, entries of indexed rows
  long long idx_reads[kWarps];        // entries read through the index
  long long cov[kWarps][4];           // coverage sums (see cover())
  int cbuf[kCtaBuf];                  // the CTA's vertices to push, moved on at the end of the phase
  int mbuf[kMemBuf];                  // the CTA's new members
  unsigned ccnt, mcnt;                // entries claimed in cbuf and mbuf (may pass their sizes)
  unsigned qn[2], qbase[4];           // the CTA's bulk push: items and units, queue, row-list and member positions
  int ok;                             // the last grid barrier did not time out
  unsigned bar;                       // arrivals the last grid barrier waited for
  Step step;                          // what the CTA does next
  Work work;
  // CTA 0 thread 0: time per phase kind, the time of the last lap, the
  // frontier sizes' sum, member-list entries in vertex order
  unsigned long long acc[4], t_last;
  long long frontiers, sorted;
};

__device__ __forceinline__ Shared& shared() {
  extern __shared__ uint4 smem_raw[];
  return *reinterpret_cast<Shared*>(smem_raw);
}
__device__ __forceinline__ Env& env() { return shared().E; }
// The counters a phase reads as its inputs.
__device__ __forceinline__ const LoopState& inputs() { return shared().snap; }

// This warp's number in the grid.
__device__ __forceinline__ unsigned team_warp() {
  return blockIdx.x * kWarps + warp_id();
}

__device__ __forceinline__ unsigned grab(unsigned* ctr) {
  unsigned x = 0;
  if (lane_id() == 0) x = atomicAdd(ctr, 1u);
  return __shfl_sync(0xffffffffu, x, 0);
}

// Smallest s <= top for which `warps` warps with 2^s of the items each take
// them all.  Shares are powers of two, found without a division.
__device__ __forceinline__ int share(unsigned items, unsigned warps, int top) {
  int s = 0;
  while (s < top && (warps << s) < items) ++s;
  return s;
}

// Hands out the work items [0, total) of a phase to warps.  Every warp's
// first 2^sh items follow from its own number; the rest are taken 2^sh at
// a time from the phase's counter (a counter takes one atomic at a time, so
// one item per atomic would bound a phase of hundreds of thousands of
// items).  2^sh grows with the items per warp (at most 32), keeping the
// tail imbalance small.  A phase of no more items than warps uses no atomic.
__device__ __forceinline__ int grab_share(unsigned items, unsigned warps) {
  int s = 0;
  while (s < 5 && (16u * warps << s) <= items) ++s;
  return s;
}
struct Grabber {
  unsigned* ctr;  // nullptr: no counter, the warps take their items in turn
  unsigned total, cur, end, base, step;
  int sh;
  __device__ __forceinline__ Grabber(unsigned* c, unsigned t, unsigned gwarp, unsigned nwarps) : ctr(c), total(t) {
    start(grab_share(t, nwarps), gwarp, nwarps);
  }
  __device__ __forceinline__ Grabber(unsigned* c, const Work& w, unsigned gwarp, unsigned nwarps) : ctr(c), total(w.total) {
    start(w.sh, gwarp, nwarps);
  }
  __device__ __forceinline__ void start(int s, unsigned gwarp, unsigned nwarps) {
    sh = s;
    step = nwarps << sh;
    base = gwarp << sh;
    cur = base;
    end = min(total, cur + (1u << sh));
  }
  // Warp-uniform.
  __device__ __forceinline__ bool next(unsigned& i) {
    if (cur >= end) {
      if (step >= total) return false;
      if (ctr) {
        cur = step + (grab(ctr) << sh);
      } else {
        base += step;
        cur = base;
      }
      if (cur >= total) {
        end = cur;
        return false;
      }
      end = min(total, cur + (1u << sh));
    }
    i = cur++;
    return true;
  }
};

// Mask words a row of L slots needs in a colour window: the mex of at most
// L colours is at most L, so colours >= min(L, kMaskBits) never matter;
// saturation sizes need the whole window.  At least 2 words (colours < 64
// are folded in from per-lane registers).
__device__ __forceinline__ int mask_words(int L, int mode) {
  if (mode == M_DISTINCT) return kMaskWords;
  const int limit = min(L, kMaskBits);
  return min(kMaskWords, max(2, (limit + 31) / 32 + 1));
}

// Work units of a row: a row of L slots pushed with unit size CH is cut
// into row_units(L, CH) units.  Consumers recover the span of every unit
// from L and the unit count alone (the queue need not record CH): the units
// split the row evenly, in multiples of 128 slots.  (Cutting hub rows into
// quarter units as well was measured 21 % slower on the headline: the extra
// units' mask combining costs more than the shorter units save.)
__device__ __forceinline__ int row_units(int L, int CH) { return L > CH ? (L + CH - 1) / CH : 1; }
__device__ __forceinline__ int unit_span(int L, int nch) {
  const int s = (L + nch - 1) / nch;
  return (s + 127) & ~127;
}

// The queue a phase's vertices go to: buffer `buf` with the counters of slot
// `q`, rows cut into units of `ch` slots.  mode: R_ROWS rows only, R_MEX with a mask region per multi-unit row,
// R_SAT the same for saturation sizes (and no class A), R_EVAL the loop's mex
// rows and R_PUSH its pushing rows (indexed rows are read through their
// index, and cut by what that reads).
enum RowMode { R_ROWS = 0, R_MEX = 1, R_SAT = 2, R_EVAL = 3, R_PUSH = 4 };
struct Target {
  short buf, q;
  int mode, ch;
  bool first;  // HI: the loop's first iteration
};

// The mask region of a multi-unit row: [done counter, mask words...], zeroed.
// -1: no room.
__device__ __forceinline__ int take_masks(const QueueBufs& qb, QCount* qc, int L, int mode, unsigned* status) {
  const unsigned words = (mask_words(L, mode == R_SAT ? M_DISTINCT : M_MEX_ALL) + 1 + 3) & ~3;
  const unsigned mo = atomicAdd(&qc->masks, words);
  if ((long long)mo + words > qb.capM) {
    atomicOr(status, ST_OVERFLOW);
    return -1;
  }
  uint4* m = reinterpret_cast<uint4*>(qb.gmask + mo);
#pragma unroll 1
  for (unsigned i = 0; i < words / 4; ++i) m[i] = make_uint4(0, 0, 0, 0);
  return (int)mo;
}

__device__ __forceinline__ void write_units(const QueueBufs& qb, unsigned at, int u, int c, int ms, unsigned* status) {
  if ((long long)at + c > qb.capU) {
    atomicOr(status, ST_OVERFLOW);
    return;
  }
#pragma unroll 1
  for (int q = 0; q < c; ++q) qb.units[at + q] = make_int4(u, q, ms, c);
}

// How a row goes into a queue: its units (0: class A) and, for a pushing
// indexed row of HI, the parts of its ordered copy and change list to walk
// (see push_parts).
struct Plan {
  int c;
  int4 parts;  // x < 0: none
};

// Writes row u of L slots at its queue positions.
__device__ __noinline__ void write_row(Target T, int u, int L, Plan P, unsigned pa, unsigned pu) {
  const Env& E = env();
  const QueueBufs& qb = E.qb[T.buf];
  QCount* qc = &E.ls->q[T.q];
  unsigned* status = &E.st->status;
  if (P.c == 0) {
    if ((long long)pa < qb.capA)
      qb.itemsA[pa] = u;
    else
      atomicOr(status, ST_OVERFLOW);
    return;
  }
  int ms = -1;
  if (T.mode == R_PUSH) {
    if (P.parts.x >= 0) {
      const unsigned mo = atomicAdd(&qc->masks, (unsigned)kPushWords);
      if ((long long)mo + kPushWords > qb.capM) {
        atomicOr(status, ST_OVERFLOW);
        return;
      }
      *reinterpret_cast<int4*>(qb.gmask + mo) = P.parts;
      ms = (int)mo;
    }
  } else if (P.c > 1 && T.mode != R_ROWS) {
    ms = take_masks(qb, qc, L, T.mode, status);
    if (ms < 0) return;
  }
  write_units(qb, pu, u, P.c, ms, status);
}

// What a pushing indexed row of HI has to walk.  v (colour cv, previous
// colour pv) can mark or dirty a neighbour u only if color[u] > pv or
// color[u] == cv: of its ordered copy the head [0, x) above pv, the segment
// [y, y + z) of colour cv where that is not in the head, and its change list,
// w entries so far.  The bounds come from the copy's bin starts.
__device__ __forceinline__ int4 push_parts(const Env& E, int v) {
  const HriBufs& H = E.hri;
  const int hi = H.hid[v];
  int4 P = make_int4(-1, 0, 0, 0);
  if (hi < 0 || hi >= H.cap_hist || inputs().hri_off != 0u) return P;
  const int xc = ld_cg(&H.xcnt[hi]);
  if ((long long)xc > H.xoff[hi + 1] - H.xoff[hi]) return P;  // its change list is incomplete
  const int* start = H.hstart + (long long)hi * kHriBins;  // entries above each colour (top bin: 0)
  const int n = (int)(H.hoff[hi + 1] - H.hoff[hi]);
  const int cv = E.g.color[v] & kColorMask, pv = E.g.prev[v];
  // the head: colours above pv (the top bin whole), and cv's own with it
  // when the colour did not change
  const int low = min(cv == pv ? cv - 1 : pv, kHriBins - 2);
  P.x = low >= 0 ? start[low] : n;
  P.y = P.x;
  if (cv < pv && cv < kHriBins - 1) {
    P.y = start[cv];
    P.z = (cv > 0 ? start[cv - 1] : n) - P.y;
  }
  P.w = xc;
  return P;
}

// Entries EVAL reads for an indexed row u of the loop: HI, its change list;
// HB, its prior neighbours, walked by one warp.  -1: no usable index.
__device__ __forceinline__ int indexed_len(const Env& E, int u) {
  const HriBufs& H = E.hri;
  if (E.hri_split) return H.hid[u] >= 0 ? 1 : -1;
  if (!E.hri_on) return -1;
  const int hi = H.hid[u];
  if (hi < 0 || hi >= H.cap_hist || inputs().hri_off != 0u) return -1;
  const int xc = ld_cg(&H.xcnt[hi]);
  return (long long)xc > H.xoff[hi + 1] - H.xoff[hi] ? -1 : xc;  // longer: the list overflowed
}

// How row u of L slots goes into T's queue.  A loop's indexed row is cut by
// what the phase reads of it.
__device__ __forceinline__ Plan plan_row(const Env& E, Target T, int u, int L) {
  Plan P;
  P.parts = make_int4(-1, 0, 0, 0);
  P.c = 0;
  if (T.mode != R_SAT && L <= kSmall) return P;
  if (E.hri.min_live > 0 && L >= E.hri.min_live) {
    if (T.mode == R_EVAL) {
      const int x = indexed_len(E, u);
      if (x >= 0) L = x;
    } else if (T.mode == R_PUSH && E.hri_on) {
      P.parts = push_parts(E, u);
      if (P.parts.x >= 0) L = P.parts.x + P.parts.z + P.parts.w;
    }
  }
  P.c = row_units(L, T.ch);
  return P;
}

// Adds 1 per calling lane (any subset of the warp) to a counter with one
// atomic; returns each lane's position.  Lanes that meet here from different
// calls may name different counters: each group takes its own.
__device__ __noinline__ unsigned take_one(unsigned* ctr) {
  const unsigned m = __match_any_sync(__activemask(), (unsigned long long)(uintptr_t)ctr);
  const int lead = __ffs(m) - 1;
  unsigned base = 0;
  if (lane_id() == lead) base = atomicAdd(ctr, (unsigned)__popc(m));
  return __shfl_sync(m, base, lead) + __popc(m & lanemask_lt());
}

__device__ __forceinline__ void write_member(const Env& E, unsigned at, int u) {
  if ((long long)at < E.mem_cap)
    E.mem[at] = u;
  else
    atomicOr(&E.st->status, ST_OVERFLOW);
}

// Pushes u (any subset of the warp calls): vertices collect in the CTA's
// buffer, which finish_push moves on at the end of the phase with one atomic
// per counter; what does not fit goes to its queue at once.  (Lanes take their
// places one by one: finding the ones that could share an atomic cost 1 - 5 %
// of a batch, 7.7 -> 7.3 ms for 96 graphs.)
__device__ __noinline__ void stage(Target T, int u) {
  Shared& sh = shared();
  const unsigned at = atomicAdd(&sh.ccnt, 1u);
  if (at < kCtaBuf) {
    sh.cbuf[at] = u;
    return;
  }
  const Env& E = sh.E;
  if (T.mode == R_EVAL) E.qb[1].itemsA[take_one(&E.ls->ev_rows[T.q - Q_EVAL])] = u;
  QCount* qc = &E.ls->q[T.q];
  const int L = E.g.len[u];
  const Plan P = plan_row(E, T, u, L);
  const unsigned pos = P.c > 0 ? atomicAdd(&qc->countU, (unsigned)P.c) : take_one(&qc->countA);
  write_row(T, u, L, P, pos, pos);
}

// u enters the frontier: the same for the end of the member list.
__device__ __noinline__ void stage_member(int u) {
  Shared& sh = shared();
  const unsigned at = atomicAdd(&sh.mcnt, 1u);
  if (at < kMemBuf)
    sh.mbuf[at] = u;
  else
    write_member(sh.E, take_one(&sh.E.ls->m_tail), u);
}

// u joins the EVAL queue, unless it is in it.
__device__ __forceinline__ void stage_eval(const Env& E, Target T, int u) {
  const unsigned bit = 1u << (u & 31);
  if (!(atomicOr(&E.inE[u >> 5], bit) & bit)) stage(T, u);
}

// Ends a phase that stages vertices, once every warp of the CTA is through.
// All threads of the CTA call it.
__device__ __noinline__ void finish_push(Target T) {
  Shared& sh = shared();
  const Env& E = sh.E;
  __syncthreads();
  const int total = min((int)sh.ccnt, kCtaBuf), members = min((int)sh.mcnt, kMemBuf);
  if (total + members == 0) return;
#pragma unroll 1
  for (int b0 = 0; b0 < max(total, members); b0 += kThreads) {
    const int i = b0 + (int)threadIdx.x;
    const int u = i < total ? sh.cbuf[i] : -1;
    const int nu = min(kThreads, max(total - b0, 0)), nm = min(kThreads, max(members - b0, 0));
    if (threadIdx.x < 2) sh.qn[threadIdx.x] = 0;
    __syncthreads();
    int L = 0;
    Plan P;
    unsigned at = 0;
    if (u >= 0) {
      L = E.g.len[u];
      P = plan_row(E, T, u, L);
      at = atomicAdd(&sh.qn[P.c == 0 ? 0 : 1], (unsigned)max(P.c, 1));
    }
    __syncthreads();
    if (threadIdx.x < 4) {
      QCount* qc = &E.ls->q[T.q];
      const int w = threadIdx.x;
      const unsigned k = w < 2 ? sh.qn[w] : w == 3 ? nm : T.mode == R_EVAL ? nu : 0;
      unsigned* ctr = w == 0 ? &qc->countA : w == 1 ? &qc->countU : w == 3 ? &E.ls->m_tail : &E.ls->ev_rows[T.q - Q_EVAL];
      if (k) sh.qbase[w] = atomicAdd(ctr, k);
    }
    __syncthreads();
    if (u >= 0) {
      // (the row list of EVAL, for the commit, is in the SCAN queue's items)
      if (T.mode == R_EVAL) E.qb[1].itemsA[sh.qbase[2] + threadIdx.x] = u;
      write_row(T, u, L, P, sh.qbase[0] + at, sh.qbase[1] + at);
    }
    if ((int)threadIdx.x < nm) write_member(E, sh.qbase[3] + threadIdx.x, sh.mbuf[i]);
    __syncthreads();
  }
  if (threadIdx.x == 0) sh.ccnt = sh.mcnt = 0;
}

// Slots per work unit for a queue pushed while processing a seeding phase of
// `items` work items with `nwarps` warps: the configured size while the
// phase keeps every warp busy, an eighth, a quarter or a half of it (at
// least 128, a multiple of 128) when it does not.
__device__ __forceinline__ int unit_slots_for(unsigned items, unsigned nwarps, int ch) {
  const int d = items < nwarps / 4 ? 8 : items < nwarps / 2 ? 4 : items < 2 * nwarps ? 2 : 1;
  const int c = (ch / d) & ~127;
  return c < 128 ? 128 : c;
}

// Numbers the slots of the lanes' rows (L slots at `at`, 0 for none) in
// the warp's table and returns their total.  All lanes must call.
__device__ __noinline__ int number_rows(Rows& R, const int* at, int L) {
  const int incl = warp_incl_scan(L);
  R.excl[lane_id()] = incl - L;
  R.at[lane_id()] = at;
  __syncwarp();
  return __shfl_sync(0xffffffffu, incl, 31);
}

// The row of slot s: the largest j with excl[j] <= s.
__device__ __forceinline__ int row_of(const Rows& R, int s) {
  int j = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1)
    if (R.excl[j + step] <= s) j += step;
  return j;
}

// First zero bit of the window sm[0..nw) (words >= nw count as zero);
// -1 when all kMaskBits bits are set.  All lanes must call.
__device__ __forceinline__ int first_zero(const unsigned* sm, int nw) {
#pragma unroll 1
  for (int k0 = 0; k0 < nw; k0 += 32) {
    const int k = k0 + lane_id();
    const unsigned word = k < nw ? sm[k] : 0u;
    const unsigned bal = __ballot_sync(0xffffffffu, word != 0xffffffffu);
    if (bal) {
      const int l = __ffs(bal) - 1;
      const unsigned wd = __shfl_sync(0xffffffffu, word, l);
      return (k0 + l) * 32 + __ffs(~wd) - 1;
    }
  }
  return nw < kMaskWords ? nw * 32 : -1;
}

// ---------------------------------------------------------------------
// slow paths (single warp, whole row): colour windows beyond the first
// ---------------------------------------------------------------------
__device__ __noinline__ int slow_mex(int v, int mode, int w_first) {
  const GraphDev& g = env().g;
  unsigned* sm = shared().mask[warp_id()];
  const long long o = g.off[v];
  const int L = g.len[v];
  const int pv = mode == M_MEX_PRIOR ? g.prop[v] : 0;
#pragma unroll 1
  for (int w0 = w_first;; w0 += kMaskBits) {
#pragma unroll 1
    for (int k = lane_id(); k < kMaskWords; k += 32) sm[k] = 0;
    __syncwarp();
#pragma unroll 1
    for (int s0 = 0; s0 < L; s0 += 32) {
      const int s = s0 + lane_id();
      if (s < L) {
        const int u = g.adj[o + s];
        if (u >= 0 && (mode != M_MEX_PRIOR || is_prior(g.prop[u], u, pv, v))) {
          const int c = (g.color[u] & kColorMask) - w0;
          if (c >= 0 && c < kMaskBits) atomicOr(&sm[c >> 5], 1u << (c & 31));
        }
      }
    }
    __syncwarp();
    const int r = first_zero(sm, kMaskWords);
    __syncwarp();
    if (r >= 0) return w0 + r;
    if (w0 > L) return w0;  // unreachable: the mex never exceeds the row length
  }
}

__device__ __noinline__ int slow_distinct(int v, int cmax) {
  const GraphDev& g = env().g;
  unsigned* sm = shared().mask[warp_id()];
  const long long o = g.off[v];
  const int L = g.len[v];
  int total = 0;
#pragma unroll 1
  for (int w0 = kMaskBits; w0 <= cmax; w0 += kMaskBits) {
#pragma unroll 1
    for (int k = lane_id(); k < kMaskWords; k += 32) sm[k] = 0;
    __syncwarp();
#pragma unroll 1
    for (int s0 = 0; s0 < L; s0 += 32) {
      const int s = s0 + lane_id();
      if (s < L) {
        const int u = g.adj[o + s];
        if (u >= 0) {
          const int c = (g.color[u] & kColorMask) - w0;
          if (c >= 0 && c < kMaskBits) atomicOr(&sm[c >> 5], 1u << (c & 31));
        }
      }
    }
    __syncwarp();
    int cnt = 0;
#pragma unroll 1
    for (int k = lane_id(); k < kMaskWords; k += 32) cnt += __popc(sm[k]);
    total += (int)warp_sum_ll(cnt);
    __syncwarp();
  }
  return total;
}

// ---------------------------------------------------------------------
// REDUCE: colour results of a queue into out[]
// ---------------------------------------------------------------------
// Folds per-lane masks of colours < 64 into words 0 and 1 of the window.
__device__ __forceinline__ void fold_low(unsigned* sm, unsigned long long lm) {
  const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)lm);
  const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(lm >> 32));
  __syncwarp();
  if (lane_id() == 0) {
    sm[0] |= lo;
    sm[1] |= hi;
  }
  __syncwarp();
}

// Combines the mask of one unit of a multi-unit row with the row's (gm[0]:
// finished units, gm[1..nw]: mask).  True for the unit that finishes last,
// whose window then holds the whole row's mask.
__device__ __forceinline__ bool merge_masks(unsigned* gm, unsigned* sm, int nw, int nch) {
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) {
    const unsigned x = sm[k];
    if (x) atomicOr(&gm[1 + k], x);
  }
  __threadfence();
  __syncwarp();
  int last = 0;
  if (lane_id() == 0) last = atomicAdd(&gm[0], 1u) == (unsigned)(nch - 1);
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return false;
  __threadfence();
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) sm[k] = ld_cg(&gm[1 + k]);
  __syncwarp();
  return true;
}

constexpr int kC8Top = 255;
__device__ __forceinline__ unsigned char to_c8(int c) { return (unsigned char)min(c, kC8Top); }

// Window bits of the colours at ids[e0..e1): four gathers in flight per
// lane (HB: of the byte colours).
template <int V>
__device__ __forceinline__ void mask_colors(const Env& E, unsigned* sm, const int* ids, long long e0, long long e1,
                                            int nbits) {
  unsigned long long lm = 0;
#pragma unroll 1
  for (long long r0 = e0; r0 < e1; r0 += 128) {
    int cc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long idx = r0 + j * 32 + lane_id();
      cc[j] = idx < e1 ? ids[idx] : -1;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = cc[j];
      if (V == DC_HB) {
        cc[j] = u >= 0 ? (int)E.c8[u] : -1;
        if (cc[j] == kC8Top) cc[j] = E.g.color[u];
      } else {
        cc[j] = u >= 0 ? (E.g.color[u] & kColorMask) : -1;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = cc[j];
      if (c < 0) continue;
      if (c < 64)
        lm |= 1ull << c;
      else if (c < nbits)
        atomicOr(&sm[c >> 5], 1u << (c & 31));
    }
  }
  fold_low(sm, lm);
}

// HI mex of an indexed row v inside the loop, from the index instead of a
// gather per neighbour: colour c is present iff some neighbour that kept
// its launch-start colour has colour c (the row's count of unchanged
// neighbours of launch-start colour c is above 0: the build counted every
// colour and the append phase takes one off for each neighbour's first
// change), or some changed neighbour has colour c now (its change list).
// Every unit of the row gathers the current colours of its slice of the
// change list into the row's mask; the unit that finishes last reads the
// counts 128 colours at a time from 0.  Returns false when the row has no
// usable index (the caller scans it).
__device__ __noinline__ bool reduce_heavy(const unsigned* gmask, int4 un, int* out) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const HriBufs& H = E.hri;
  const int v = un.x;
  const int L = E.g.len[v];
  const int xc = L >= H.min_live ? indexed_len(E, v) : -1;
  if (xc < 0) return false;
  const int hi = H.hid[v];
  const long long xb = H.xoff[hi];
  const int nch = un.w;
  const int nw = mask_words(L, M_MEX_ALL);  // as the queue push sized the row's mask
  unsigned* sm = sh.mask[warp_id()];
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) sm[k] = 0;
  __syncwarp();
  const int us = unit_span(xc, nch);
  const long long e0 = (long long)un.y * us;
  const long long e1 = min((long long)xc, e0 + us);
  mask_colors<DC_HI>(E, sm, H.xv + xb, e0, e1, nw * 32);
  if (lane_id() == 0 && e1 > e0) sh.idx_reads[warp_id()] += e1 - e0;
  if (nch > 1 && !merge_masks(const_cast<unsigned*>(gmask) + un.z, sm, nw, nch)) return true;
  const int* cnt = H.hist + (long long)hi * kHriBins;
  int r = -1;
#pragma unroll 1
  for (int c0 = 0; c0 < kHriBins - 1 && r < 0; c0 += 128) {
    int n4[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = c0 + j * 32 + lane_id();
      n4[j] = c < kHriBins - 1 ? ld_cg(&cnt[c]) : 1;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = c0 + j * 32 + lane_id();
      const bool pres = n4[j] > 0 || (c < nw * 32 && ((sm[c >> 5] >> (c & 31)) & 1u));
      const unsigned bal = __ballot_sync(0xffffffffu, pres);
      if (r < 0 && bal != 0xffffffffu) r = c0 + j * 32 + __ffs(~bal) - 1;
    }
  }
  if (r < 0) {
    // every colour below the shared top bin is present: scan the row
    if (lane_id() == 0) sh.idx_reads[warp_id()] += L;
    r = slow_mex(v, M_MEX_ALL, 0);
  }
  if (lane_id() == 0) out[v] = r;
  __syncwarp();
  return true;
}

// HB mex over the prior neighbours of an indexed row v (seeding and loop):
// only the first hsplit entries of its copy are prior to v, so only their
// colours are gathered.  The whole row is handled by its first unit.
__device__ __noinline__ bool reduce_split(int4 un, bool loop, int* out) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const HriBufs& H = E.hri;
  const int v = un.x;
  const int hi = E.g.len[v] >= H.min_live ? H.hid[v] : -1;
  if (hi < 0) return false;
  if (un.y != 0) return true;
  const long long pb = H.hoff[hi];
  const int nh = H.hsplit[hi];
  unsigned* sm = sh.mask[warp_id()];
  const int nw = mask_words(nh + 1, M_MEX_ALL);  // the mex of nh colours is at most nh
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) sm[k] = 0;
  __syncwarp();
  mask_colors<DC_HB>(E, sm, H.ids + pb, 0, nh, nw * 32);
  int r = first_zero(sm, nw);
  __syncwarp();
  if (r < 0) r = slow_mex(v, M_MEX_PRIOR, kMaskBits);  // every colour of the window present
  if (lane_id() == 0) {
    out[v] = r;
    sh.idx_reads[warp_id()] += nh;
    if (!loop) {
      const long long live = H.hoff[hi + 1] - pb;  // the rule covers every live entry
      sh.scanned[warp_id()] += live;
      sh.idx_cov[warp_id()] += live;
    }
  }
  __syncwarp();
  return true;
}

template <int V>
__device__ __noinline__ void reduce_unit(int4 un, const unsigned* gmask, int mode, bool loop, int* out) {
  Shared& sh = shared();
  const Env& E = sh.E;
  if (V == DC_HI && loop && E.hri_on && reduce_heavy(gmask, un, out)) return;
  if (V == DC_HB && E.hri_split && reduce_split(un, loop, out)) return;
  const int* color = E.g.color;
  const unsigned long long* cp = E.cp;
  const int v = un.x, chunk = un.y, nch = un.w;
  const int L = E.g.len[v];
  const int* adj = E.g.adj + E.g.off[v];
  const int us = unit_span(L, nch);
  const int s_lo = chunk * us;
  const int s_hi = min(L, s_lo + us);
  const int limit = mode == M_DISTINCT ? kMaskBits : min(L, kMaskBits);
  const int nw = mask_words(L, mode);
  unsigned* sm = sh.mask[warp_id()];
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) sm[k] = 0;
  __syncwarp();
  const int pv = V == DC_HB ? E.g.prop[v] : 0;
  unsigned long long lm = 0;  // colours < 64 seen by this lane
  int seen = 0;
  // Four slots per lane per round, lane l taking slots r0 + l + 32 j: every
  // load is coalesced across the warp, and because rows are kept sorted by
  // neighbour id, the colour gathers of one instruction fall on nearby
  // addresses in dense rows.  Four independent gathers are in flight.
  // The ids of round r + 1 are loaded before the colour gathers of round r
  // are consumed, so each round waits on one dependent load, not two.
  int nx[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int sidx = s_lo + j * 32 + lane_id();
    nx[j] = sidx < s_hi ? __ldg(adj + sidx) : -1;
  }
#pragma unroll 1
  for (int r0 = s_lo; r0 < s_hi; r0 += 128) {
    int uu[4], cc[4], pp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uu[j] = nx[j];
      const int sidx = r0 + 128 + j * 32 + lane_id();
      nx[j] = sidx < s_hi ? __ldg(adj + sidx) : -1;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (V == DC_HB) {
        const unsigned long long x = uu[j] >= 0 ? cp[uu[j]] : 0ull;
        cc[j] = (int)((unsigned)x & (unsigned)kColorMask);
        pp[j] = (int)(x >> 32);
      } else {
        cc[j] = uu[j] >= 0 ? (color[uu[j]] & kColorMask) : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (uu[j] < 0) continue;
      ++seen;
      if (V == DC_HB && !is_prior(pp[j], uu[j], pv, v)) continue;
      const int c = cc[j];
      if (c < 64)
        lm |= 1ull << c;
      else if (c < limit)
        atomicOr(&sm[c >> 5], 1u << (c & 31));
    }
  }
  fold_low(sm, lm);
  if (!loop) {
    seen = __reduce_add_sync(0xffffffffu, seen);
    if (lane_id() == 0) sh.scanned[warp_id()] += seen;
  }
  if (nch > 1 && !merge_masks(const_cast<unsigned*>(gmask) + un.z, sm, nw, nch)) return;
  int r;
  if (V == DC_HI && mode == M_DISTINCT) {
    int cnt = 0;
#pragma unroll 1
    for (int k = lane_id(); k < nw; k += 32) cnt += __popc(sm[k]);
    r = __reduce_add_sync(0xffffffffu, cnt);
    __syncwarp();
    const int cmax = ld_cg(&E.st->cmax);
    if (cmax >= kMaskBits) r += slow_distinct(v, cmax);
  } else {
    r = first_zero(sm, nw);
    __syncwarp();
    if (r < 0) r = slow_mex(v, mode, kMaskBits);
  }
  if (lane_id() == 0) out[v] = r;
  __syncwarp();
}

// Class A batch: 32 rows of <= kSmall slots.  MEX modes only.  Each lane
// handles four slots per round, so four gathers are in flight.
template <int V>
__device__ __noinline__ void reduce_batchA(const int* items, unsigned cA, unsigned idx, bool loop, int* out) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const int* color = E.g.color;
  const bool valid = idx < cA;
  const int v = valid ? items[idx] : 0;
  const int L = valid ? E.g.len[v] : 0;
  const int* at = E.g.adj + (valid ? E.g.off[v] : 0);
  Rows& R = sh.rows[warp_id()];
  unsigned long long* m64 = reinterpret_cast<unsigned long long*>(sh.mask[warp_id()]);
  m64[lane_id()] = 0ull;
  if (V == DC_HB) {
    R.a[lane_id()] = v;
    R.b[lane_id()] = valid ? E.g.prop[v] : 0;
  }
  const int T = number_rows(R, at, L);
  int seen = 0;
#pragma unroll 1
  for (int s0 = lane_id(); s0 < T; s0 += 128) {
    int jj[4], uu[4], cc[4], pp[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * 32;
      jj[r] = row_of(R, s);
      uu[r] = s < T ? R.at[jj[r]][s - R.excl[jj[r]]] : -1;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (V == DC_HB) {
        const unsigned long long x = uu[r] >= 0 ? E.cp[uu[r]] : 0ull;
        cc[r] = (int)((unsigned)x & (unsigned)kColorMask);
        pp[r] = (int)(x >> 32);
      } else {
        cc[r] = uu[r] >= 0 ? (color[uu[r]] & kColorMask) : 0;
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (uu[r] < 0) continue;
      ++seen;
      if (V == DC_HB && !is_prior(pp[r], uu[r], R.b[jj[r]], R.a[jj[r]])) continue;
      if (cc[r] < 64) atomicOr(reinterpret_cast<unsigned*>(&m64[jj[r]]) + (cc[r] >> 5), 1u << (cc[r] & 31));
    }
  }
  __syncwarp();
  if (valid) out[v] = __ffsll((long long)~m64[lane_id()]) - 1;
  if (!loop) {
    seen = __reduce_add_sync(0xffffffffu, seen);
    if (lane_id() == 0) sh.scanned[warp_id()] += seen;
  }
  __syncwarp();
}

// Rows of a class-A batch: 32 when there are rows for every warp, fewer when
// that leaves warps without work (a batch of 32 rows of 32 slots is eight
// dependent rounds for its warp, one of four rows is one).  Lanes past the
// batch's rows get an index past the queue.
__device__ __forceinline__ int batch_share(unsigned cA, unsigned cU, unsigned nwarps) {
  return share(cA, nwarps > 2 * cU ? nwarps - cU : nwarps / 2, 5);
}
__device__ __forceinline__ unsigned shares(unsigned items, int s) { return (items + (1u << s) - 1) >> s; }
// Pieces a phase's units are walked in: a unit of the loop is kLoopUnit slots
// (four rounds of a warp's walk); while there are idle warps, each round
// gets a warp of its own.
__device__ __forceinline__ int unit_pieces(unsigned units, unsigned nwarps) {  // log2
  return units <= nwarps / 2 ? 2 : units <= nwarps ? 1 : 0;
}
__device__ __forceinline__ unsigned batch_item(unsigned b, int s) {
  return lane_id() < (1 << s) ? (b << s) + lane_id() : 0xffffffffu;
}

template <int V>
__device__ __noinline__ void phase_reduce(int buf, int q, unsigned* ctr, int mode, bool loop, int* out) {
  const Env& E = env();
  const QueueBufs& qb = E.qb[buf];
  const QCount& qc = inputs().q[q];
  const unsigned cA = (unsigned)min((long long)qc.countA, qb.capA);
  const unsigned cU = (unsigned)min((long long)qc.countU, qb.capU);
  const int per = batch_share(cA, cU, E.nwarps);
  Grabber gb(ctr, cU + shares(cA, per), team_warp(), E.nwarps);
  unsigned i;
#pragma unroll 1
  while (gb.next(i)) {
    if (i < cU)
      reduce_unit<V>(qb.units[i], qb.gmask, mode, loop, out);
    else
      reduce_batchA<V>(qb.itemsA, cA, batch_item(i - cU, per), loop, out);
  }
}

// The word that holds u's frontier flags: its colour word (HI) or the colour
// half of its packed word (HB).
template <int V>
__device__ __forceinline__ unsigned* flag_word(const Env& E, int u) {
  return V == DC_HB ? reinterpret_cast<unsigned*>(E.cp + u) : reinterpret_cast<unsigned*>(E.g.color + u);
}

__device__ __forceinline__ bool in_bits(const unsigned* bm, int v) { return (bm[v >> 5] >> (v & 31)) & 1u; }
__device__ __forceinline__ void set_bit(unsigned* bm, int v) { atomicOr(&bm[v >> 5], 1u << (v & 31)); }
__device__ __forceinline__ void clear_bit(unsigned* bm, int v) { atomicAnd(&bm[v >> 5], ~(1u << (v & 31))); }

// Index of u's heavy row, or -1.  Checked against the row list, because a
// pool launch indexes its own graphs' rows only and the entries of other
// vertices are left from earlier launches.
__device__ __noinline__ int heavy_row(int u) {
  const Env& E = env();
  const int hi = E.hri.hid[u];
  if (hi < 0 || hi >= E.hri.cap_rows || (unsigned long long)hi >= ld_cg(&E.st->hcount)) return -1;
  return E.hri.hrow[hi] == u ? hi : -1;
}

// ---------------------------------------------------------------------
// PUSH: findEligibleNeighbors from the frontier vertices that are new or
// (HI) changed, and dirty marks from the ones whose colour changed
//   HI: HI/gpuFunctions_undir.cuh:229-260
//   HB: HB/gpuFunctions_undir.cuh:259-291
// ---------------------------------------------------------------------
// HB keeps "entered the frontier with the last commit" in bit 30 of prev[v].
constexpr int kNewBit = 1 << 30;

struct Rule {
  int v, cv, pv;  // pushing vertex, its colour, its colour before the last commit (HB: and kNewBit)
  int pr;         // HB: degree property
};

template <int V>
__device__ __forceinline__ Rule rule_of(const Env& E, int v) {
  Rule R;
  R.v = v;
  R.pv = E.g.prev[v];
  R.cv = E.g.color[v] & kColorMask;
  R.pr = V == DC_HB ? E.g.prop[v] : 0;
  return R;
}

// Applies four candidates per lane at once (their gathers and atomics are in
// flight together).  The entry (v -> u) marks u for the next frontier (HI:
// v's previous colour is below u's, or they share a colour and v < u; HB: v
// is new, u being a neighbour v is prior to) and makes u dirty when v
// changed, leaving a colour below u's or taking u's.  A marked vertex
// outside the frontier is claimed through the mark bit of its word, joins the
// member list with v as its witness, and has its mex computed; a marked
// member of the first frontier (HI) gets its first witness (later on members
// keep the one they have: a changed v is a short-lived witness, and replacing
// good ones by it took 20 % more time at R-MAT scale 24); a dirty vertex
// loses its clean bit, and
// the warp that took it queues the vertex for its mex: it is in the next
// frontier, because v marks it (HB: v is a frontier vertex prior to u; HI:
// unless they share a colour and u < v, where u changed in the same commit,
// and members that changed are queued by PULL if they stay).  ww: u's colour
// word.
template <int V>
__device__ __forceinline__ void push4(const Env& E, Target T, const Rule* R, const int* uu, const unsigned* ww) {
  unsigned old[4], cw[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int cu = (int)(ww[j] & (unsigned)kColorMask);
    const int pv = V == DC_HB ? (R[j].pv & kColorMask) : R[j].pv;
    const bool in = uu[j] >= 0;
    const bool low = pv < cu, same = R[j].cv == cu;
    const bool dirty = in && pv != R[j].cv && (low || same);
    const bool mark = in && (V == DC_HI ? low || (same && R[j].v < uu[j]) : (R[j].pv & kNewBit) != 0);
    old[j] = kMarkBit;
    cw[j] = dirty ? E.clean[uu[j] >> 5] : 0u;
    if (V == DC_HI && !mark) cw[j] &= ~(1u << (uu[j] & 31));
    if (mark) {
      if (ww[j] & kInF) {
        if (V == DC_HI && T.first) E.wit[uu[j]] = R[j].v;
      } else if (!(ww[j] & kMarkBit)) {
        old[j] = atomicOr(flag_word<V>(E, uu[j]), kMarkBit);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned bit = 1u << (uu[j] & 31);
    bool eval = false;
    if (cw[j] & bit) eval = (atomicAnd(&E.clean[uu[j] >> 5], ~bit) & bit) != 0u;
    if (!(old[j] & kMarkBit)) {
      E.wit[uu[j]] = R[j].v;
      if (V == DC_HI && E.gcount) atomicAdd(&E.gcount[E.gid[uu[j]]], 1);
      stage_member(uu[j]);
      eval = true;
    }
    if (eval) stage_eval(E, T, uu[j]);
  }
}

// HB: dirty marks of an indexed row's changed vertex that marks no one (it
// was a member before its last commit), over ids[lo..top) of the neighbours
// behind it.  Nine in ten entries fail the test on the colour, and nearly all
// that pass are dirty already, so the walk is its gathers, and these are
// bound by the cache lines a warp's 32 lanes touch (one a clock per SM; about
// 23 of 128 vertices each at R-MAT scale 22).  Byte colours need fewer and
// more often hit the L1 than the packed words: 62 M entries in 190 us where
// the packed words took 219, the whole batch 80.0 -> 75.7 ms.  (Ordering the
// rows by launch-start colour leaves 17 % of the entries, but with change
// lists that hold most neighbours after 20 iterations nothing is saved;
// ordering them by how many neighbours come before each, which bounds its
// colour, leaves 80 %.)
__device__ __noinline__ void push_dirty(Target T, const int* ids, int lo, int top, int pv, int cv) {
  const Env& E = env();
  const unsigned char* c8 = E.c8;
  constexpr int U = 4;
  int nx[U];
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const int i = lo + j * 32 + lane_id();
    nx[j] = i < top ? __ldcg(ids + i) : -1;
  }
#pragma unroll 1
  for (int r0 = lo; r0 < top; r0 += 32 * U) {
    int uu[U], cc[U];
    bool any = false;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      uu[j] = nx[j];
      const int i = r0 + 32 * U + j * 32 + lane_id();
      nx[j] = i < top ? __ldcg(ids + i) : -1;
    }
#pragma unroll
    for (int j = 0; j < U; ++j) cc[j] = uu[j] >= 0 ? (int)c8[uu[j]] : -1;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (uu[j] < 0 || !(cc[j] > pv || cc[j] == cv || cc[j] == kC8Top)) uu[j] = -1;
      any |= uu[j] >= 0;
    }
    if (!__any_sync(0xffffffffu, any)) continue;
    unsigned cw[U];
#pragma unroll
    for (int j = 0; j < U; ++j) cw[j] = uu[j] >= 0 ? E.clean[uu[j] >> 5] : 0u;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const unsigned bit = 1u << (uu[j] & 31);
      if (!(cw[j] & bit)) continue;
      if (cc[j] == kC8Top) {
        const int cu = E.g.color[uu[j]];
        if (!(pv < cu || cv == cu)) continue;
      }
      if (atomicAnd(&E.clean[uu[j] >> 5], ~bit) & bit) stage_eval(E, T, uu[j]);
    }
    __syncwarp();
  }
}

// PUSH over piece `sub` of `pieces` of one unit of a row: its neighbours, or,
// of an indexed row, HI: the parts of its ordered copy and its change list
// that push_parts named; HB: the part of its copy behind the prior
// neighbours.  Every candidate's current colour is gathered and the rule
// applied to it.
template <int V>
__device__ __noinline__ void push_unit(Target T, int4 un, const unsigned* gmask, int sub, int pieces) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const int v = un.x;
  if (V == DC_HB && E.gskip && ld_cg(&E.gskip[E.gid[v]]) == 0) return;  // its graph has stopped
  const int L = E.g.len[v];
  bool indexed = false;
  int n = L;           // entries the row's units share
  int4 P;              // HI, indexed: the parts
  P.x = P.y = P.z = 0;
  const int* ids = E.g.adj + E.g.off[v];
  const unsigned long long* pairs = nullptr;
  Rule R[4];
  R[0] = R[1] = R[2] = R[3] = rule_of<V>(E, v);
  int total = L;
  if (V == DC_HI && un.z >= 0 && inputs().hri_off == 0u) {
    indexed = true;
    P = ld_cg(reinterpret_cast<const int4*>(gmask + un.z));
    const int hi = E.hri.hid[v];
    pairs = E.hri.pairs + E.hri.hoff[hi];
    ids = E.hri.xv + E.hri.xoff[hi];
    n = P.x + P.z + P.w;
    // the list may have grown since the row was cut: the last piece goes on
    total = P.x + P.z + ld_cg(&E.hri.xcnt[hi]);
  } else if (V == DC_HB && E.hri_split && L >= E.hri.min_live) {
    const int hi = heavy_row(v);
    if (hi >= 0) {
      indexed = true;
      const long long b = E.hri.hoff[hi] + E.hri.hsplit[hi];
      ids = E.hri.ids + b;
      total = n = (int)(E.hri.hoff[hi + 1] - b);
    }
  }
  const int us = unit_span(n, un.w * pieces), piece = un.y * pieces + sub;
  const int lo = piece * us;
  const int top = piece == un.w * pieces - 1 ? total : min(total, lo + us);
  if (V == DC_HB && indexed && !(R[0].pv & kNewBit)) {
    if (R[0].pv != R[0].cv) push_dirty(T, ids, lo, top, R[0].pv, R[0].cv);
    if (lane_id() == 0 && lo < top) sh.idx_reads[warp_id()] += top - lo;
    return;
  }
  const int np = P.x + P.z;  // entries in the ordered copy
  const int* color = E.g.color;
  // the ids of round r0 + 128 are loaded before round r0's are consumed
  int nx[4] = {-1, -1, -1, -1};
#pragma unroll 1
  for (int r0 = lo - 128; r0 < top; r0 += 128) {
    int uu[4];
    unsigned ww[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uu[j] = nx[j];
      const int i = r0 + 128 + j * 32 + lane_id();
      nx[j] = -1;
      if (i < top) {
        if (V == DC_HI && pairs && i < np)
          nx[j] = (int)(unsigned)pairs[i < P.x ? i : P.y + (i - P.x)];
        else
          nx[j] = ids[V == DC_HI && pairs ? i - np : i];
      }
    }
    if (r0 < lo) continue;
    // one gather gives u's colour and its frontier flags (HB: and its degree
    // property, where the entries are not known to be behind v)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (V == DC_HB && !indexed) {
        const unsigned long long x = uu[j] >= 0 ? E.cp[uu[j]] : 0ull;
        ww[j] = (unsigned)x;
        if (uu[j] >= 0 && !is_prior(R[0].pr, v, (int)(x >> 32), uu[j])) uu[j] = -1;
      } else {
        ww[j] = uu[j] < 0 ? 0u : V == DC_HB ? *flag_word<V>(E, uu[j]) : (unsigned)color[uu[j]];
      }
    }
    push4<V>(E, T, R, uu, ww);
    __syncwarp();
  }
  if (indexed && lane_id() == 0 && lo < top) sh.idx_reads[warp_id()] += top - lo;
}

// Class A batch: 32 rows of <= kSmall slots, four slots per lane per round.
template <int V>
__device__ __noinline__ void push_batchA(Target T, const int* items, unsigned cA, unsigned idx) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const int* color = E.g.color;
  bool valid = idx < cA;
  const int v = valid ? items[idx] : 0;
  if (V == DC_HB && valid && E.gskip && ld_cg(&E.gskip[E.gid[v]]) == 0) valid = false;  // its graph has stopped
  Rows& W = sh.rows[warp_id()];
  int L = 0;
  const int* at = E.g.adj;
  if (valid) {
    const Rule M = rule_of<V>(E, v);
    W.a[lane_id()] = v;
    W.b[lane_id()] = M.cv;
    W.c[lane_id()] = M.pv;
    if (V == DC_HB) W.d[lane_id()] = M.pr;
    L = E.g.len[v];
    at += E.g.off[v];
  }
  const int total = number_rows(W, at, L);
#pragma unroll 1
  for (int s0 = lane_id(); s0 < total; s0 += 128) {
    Rule R[4];
    int uu[4];
    unsigned ww[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * 32;
      const int j = row_of(W, s);
      uu[r] = s < total ? W.at[j][s - W.excl[j]] : -1;
      R[r].v = W.a[j];
      R[r].cv = W.b[j];
      R[r].pv = W.c[j];
      R[r].pr = V == DC_HB ? W.d[j] : 0;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (V == DC_HB) {
        const unsigned long long x = uu[r] >= 0 ? E.cp[uu[r]] : 0ull;
        ww[r] = (unsigned)x;
        if (uu[r] >= 0 && !is_prior(R[r].pr, R[r].v, (int)(x >> 32), uu[r])) uu[r] = -1;
      } else {
        ww[r] = uu[r] >= 0 ? (unsigned)color[uu[r]] : 0u;
      }
    }
    push4<V>(E, T, R, uu, ww);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------
// PULL: which members stay
// ---------------------------------------------------------------------
constexpr int kScanUnit = 512;    // longer rows than a warp searches inline go on in units of this


// The entries of u's row that can keep it in the frontier: all of them, or
// (HB) the prior part of an indexed row.
struct Span {
  const int* at;
  int len;
  bool prior;  // every entry is prior to u
};

template <int V>
__device__ __forceinline__ Span span_of(const Env& E, int u) {
  Span s;
  if (V == DC_HB && E.hri_split) {
    const int hi = heavy_row(u);
    if (hi >= 0) {
      s.at = E.hri.ids + E.hri.hoff[hi];
      s.len = E.hri.hsplit[hi];
      s.prior = true;
      return s;
    }
  }
  s.at = E.g.adj + E.g.off[u];
  s.len = E.g.len[u];
  s.prior = false;
  return s;
}

// Which of four neighbours keep their members in the next frontier: k = 0
// no, 1 as a frontier vertex that marks the member, 2 (HB) because its
// colour equals the member's.  x < 0: none.  Member i is u[i] with colour
// c[i] and (HB) degree property p[i]; pr[i]: every entry of its span is
// prior to it.  The gathers of one kind are all in flight together (taken
// one neighbour at a time, the branches between them made each round of the
// search a chain of as many dependent round trips).
template <int V>
__device__ __forceinline__ void keeps4(const Env& E, const int* x, const int* u, const int* c, const int* p,
                                       const bool* pr, int* k) {
  if (V == DC_HI) {
    int cx[4], px[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned word = x[i] >= 0 ? E.inF[x[i] >> 5] : 0u;
      k[i] = (int)((word >> (x[i] & 31)) & 1u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      cx[i] = k[i] ? E.g.color[x[i]] : 0;
      px[i] = k[i] ? E.g.prev[x[i]] : 0;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      k[i] = k[i] && (px[i] < c[i] || ((cx[i] & kColorMask) == c[i] && x[i] < u[i])) ? 1 : 0;
  } else {
    unsigned long long xx[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) xx[i] = x[i] >= 0 ? E.cp[x[i]] : 0ull;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool pri = x[i] >= 0 && (pr[i] || is_prior((int)(xx[i] >> 32), x[i], p[i], u[i]));
      k[i] = !pri ? 0 : ((unsigned)xx[i] & kInF) ? 1 : (int)((unsigned)xx[i] & (unsigned)kColorMask) == c[i] ? 2 : 0;
    }
  }
}

// Looks for a reason to keep member u in entries [s_lo, s_hi) of its span,
// the whole warp together, 128 entries a round; ends at the first hit (whose
// witness is stored).
template <int V>
__device__ __noinline__ bool scan_span(const int* at, int s_lo, int s_hi, int u, int cu, int pu, bool prior) {
  const Env& E = env();
  const int uu[4] = {u, u, u, u}, cc[4] = {cu, cu, cu, cu}, pp[4] = {pu, pu, pu, pu};
  const bool rr[4] = {prior, prior, prior, prior};
  int nx[4] = {-1, -1, -1, -1};
#pragma unroll 1
  for (int s0 = s_lo - 128; s0 < s_hi; s0 += 128) {
    int x[4], kk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[j] = nx[j];
      const int s = s0 + 128 + j * 32 + lane_id();
      nx[j] = s < s_hi ? at[s] : -1;
    }
    if (s0 < s_lo) continue;
    keeps4<V>(E, x, uu, cc, pp, rr, kk);
    int k = 0, w = -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (kk[j] == 1) w = x[j];
      k |= kk[j];
    }
    if (__any_sync(0xffffffffu, k != 0)) {
      if (w >= 0) E.wit[u] = w;
      return true;
    }
  }
  return false;
}

constexpr int kNoWitness = -2;  // witness of a vertex that left

enum Outcome { O_NONE = 0, O_STAY = 1, O_LEAVE = 2, O_STOPPED = 3 };

// Cuts a long span of u (place `at` in the member list) from entry `from` on
// into SCAN units.
__device__ __noinline__ void push_scan(int u, int from, int len, unsigned at) {
  const Env& E = env();
  const QueueBufs& sq = E.qb[1];
  QCount* sc = &E.ls->q[Q_SCAN];
  const int c = (len - from + kScanUnit - 1) / kScanUnit;
  const unsigned mo = atomicAdd(&sc->masks, (unsigned)kScanWords);
  const unsigned pu = atomicAdd(&sc->countU, (unsigned)c);
  if ((long long)mo + kScanWords > sq.capM) {
    atomicOr(&E.st->status, ST_OVERFLOW);
    return;
  }
  // [0] finished pieces, [1] hit, [2] place in the member list, [3] first entry
  *reinterpret_cast<uint4*>(sq.gmask + mo) = make_uint4(0, 0, at, (unsigned)from);
  write_units(sq, pu, u, c, (int)mo, &E.st->status);
}

// Witness search of the lanes with need set: rows of up to kScanBatch
// entries 32 at a time (four slots per lane), the first `inl` entries of
// longer ones one row at a time with the whole warp; what is longer without
// a hit goes on in units of the SCAN queue (outcome O_NONE until that phase
// settles it).  Returns each lane's outcome.  All lanes must call.
template <int V>
__device__ __noinline__ int find_witness(bool need, int u, int cu, unsigned at, int inl) {
  Shared& sh = shared();
  const Env& E = sh.E;
  Rows& T = sh.rows[warp_id()];
  Span sp;
  sp.at = nullptr;
  sp.len = 0;
  sp.prior = false;
  if (need) {
    sp = span_of<V>(E, u);
    T.a[lane_id()] = u;
    T.b[lane_id()] = cu;
    if (V == DC_HB) T.c[lane_id()] = E.g.prop[u];
  }
  const bool shrt = need && sp.len <= kScanBatch;
  // -1: not found, 0: (HB) kept by an equal colour, else the witness + 1;
  // bit 30 on a length marks a span of prior entries only
  T.d[lane_id()] = -1;
  const int total = number_rows(T, sp.at, shrt ? sp.len : 0);
  const unsigned priors = __ballot_sync(0xffffffffu, sp.prior);
#pragma unroll 1
  for (int s0 = lane_id(); s0 < total; s0 += 128) {
    int jj[4], xx[4], kk[4], uj[4], cj[4], pj[4];
    bool pr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * 32;
      const int j = row_of(T, s);
      jj[r] = j;
      xx[r] = s < total ? T.at[j][s - T.excl[j]] : -1;
      uj[r] = T.a[j];
      cj[r] = T.b[j];
      pj[r] = V == DC_HB ? T.c[j] : 0;
      pr[r] = V == DC_HB && ((priors >> j) & 1u);
    }
    keeps4<V>(E, xx, uj, cj, pj, pr, kk);
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (kk[r] != 0) atomicMax(&T.d[jj[r]], kk[r] == 1 ? xx[r] + 1 : 0);
  }
  __syncwarp();
  const int f = T.d[lane_id()];
  bool hit = shrt && f >= 0;
  if (hit && f > 0) E.wit[u] = f - 1;
  // longer rows; their lengths in place of the slot numbers
  __syncwarp();
  T.excl[lane_id()] = sp.len;
  __syncwarp();
  unsigned todo = __ballot_sync(0xffffffffu, need && !shrt && inl > 0);
#pragma unroll 1
  while (todo) {
    const int l = __ffs(todo) - 1;
    todo &= todo - 1;
    const bool h = scan_span<V>(T.at[l], 0, min(T.excl[l], inl), T.a[l], T.b[l], V == DC_HB ? T.c[l] : 0, (priors >> l) & 1u);
    if (lane_id() == l) hit = h;
  }
  const bool lng = need && !shrt && !hit && sp.len > inl;
  if (lng) push_scan(u, inl, sp.len, at);
  __syncwarp();
  return !need || lng ? O_NONE : hit ? O_STAY : O_LEAVE;
}

// Sum of a non-negative int per lane.
__device__ __noinline__ long long warp_sum_u(int x) {
  return (long long)__reduce_add_sync(0xffffffffu, (unsigned)x & 0xffffu) +
         ((long long)__reduce_add_sync(0xffffffffu, (unsigned)x >> 16) << 16);
}

// Coverage of the loop's rules (dc_stats.slots_scanned): an iteration covers
// the rows of the frontier it starts from and of the one it finds.  A vertex
// that enters with iteration e and leaves with iteration l counts 2 (l - e)
// times, one that stays to the end T counts 2 (T - e) + 1 times, so it is
// enough to add live * -2 e on entry and live * 2 l on leaving, and the
// live entries of the last frontier 2 T + 1 times: c[0] the weighted sum,
// c[1] the entries of the current members, c[2], c[3] the same for indexed
// rows.  All lanes must call; lv: the vertex's live entries (0: none).
__device__ __noinline__ void cover(int lv, bool enter, long long weight) {
  Shared& sh = shared();
  const bool idx = (sh.E.hri_on || sh.E.hri_split) && lv >= sh.E.hri.min_live;  // long enough for the index
  const long long all = warp_sum_u(lv), ind = warp_sum_u(idx ? lv : 0);
  if (lane_id() == 0) {
    long long* c = sh.cov[warp_id()];
    c[0] += weight * all;
    c[1] += enter ? all : -all;
    c[2] += weight * ind;
    c[3] += enter ? ind : -ind;
  }
}

// Settles one member per lane: one that stays has its mex computed if it may
// have changed for a reason PUSH does not see (`eval`: HI, its own colour
// changed in the last commit; first iteration, never computed), one that
// leaves goes to the commit's list and gets no witness, so that the commit
// drops a mex computed for it: a member that goes on to SCAN (`scan`) joins
// the EVAL queue before it is known to stay.  `at` is u's place in the member
// list.  All lanes must call.
template <int V>
__device__ __noinline__ void settle(Target T, int it, int ring, int oc, int u, unsigned at, bool eval,
                                    bool scan) {
  const Env& E = env();
  const bool gone = oc == O_LEAVE || oc == O_STOPPED;
  if ((oc == O_STAY || scan) && eval) stage_eval(E, T, u);
  __syncwarp();
  const unsigned bg = __ballot_sync(0xffffffffu, gone);
  if (!bg) return;
  unsigned base = 0;
  if (lane_id() == 0) base = atomicAdd(&E.ls->m_out[ring], (unsigned)__popc(bg));
  base = __shfl_sync(0xffffffffu, base, 0) + __popc(bg & lanemask_lt());
  int lv = 0;
  if (gone) {
    E.mout[base] = u;
    E.mem[at] = -1;
    E.wit[u] = kNoWitness;
    lv = E.g.live[u];
    if (V == DC_HI && E.gcount) atomicAdd(&E.gcount[E.gid[u]], -1);
  }
  cover(oc == O_LEAVE ? lv : 0, false, 2ll * it);
  // a stopped graph's rows are not covered by the iteration they leave with
  if (V == DC_HB && __any_sync(0xffffffffu, oc == O_STOPPED)) cover(oc == O_STOPPED ? lv : 0, false, 2ll * it - 1);
}

// PULL over one piece of the member list, `m` entries from b0 on (W of 32 at
// a time, their loads in flight together).
template <int V, int W>
__device__ __noinline__ void pull_members(Target T, int it, int ring, unsigned b0, unsigned m, unsigned len,
                                          int inl) {
  const Env& E = env();
  int u[W], w[W], cu[W];
  bool eval[W], fw[W];
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const unsigned k = j * 32 + lane_id();
    u[j] = k < m && b0 + k < len ? E.mem[b0 + k] : -1;
  }
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const bool on = u[j] >= 0;
    w[j] = on ? E.wit[u[j]] : -1;
    cu[j] = V == DC_HI && on ? (E.g.color[u[j]] & kColorMask) : 0;
    eval[j] = V == DC_HI && on && E.g.prev[u[j]] != cu[j];
  }
#pragma unroll
  for (int j = 0; j < W; ++j) fw[j] = w[j] >= 0 && in_bits(E.inF, w[j]);
  if (V == DC_HI) {
    int cw[W], pw[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
      cw[j] = w[j] >= 0 ? (E.g.color[w[j]] & kColorMask) : 0;
      pw[j] = w[j] >= 0 ? E.g.prev[w[j]] : 0;
    }
#pragma unroll
    for (int j = 0; j < W; ++j) fw[j] = fw[j] && (pw[j] < cu[j] || (cw[j] == cu[j] && w[j] < u[j]));
  }
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const unsigned i = b0 + j * 32 + lane_id();
    int oc = O_NONE;
    if (u[j] >= 0) {
      if (V == DC_HB && E.gskip && ld_cg(&E.gskip[E.gid[u[j]]]) == 0)
        oc = O_STOPPED;
      else if (fw[j])
        oc = O_STAY;
      else if (V == DC_HI && it == 1 && w[j] < 0)
        oc = O_LEAVE;  // all of the first frontier has pushed: nothing marked u
      if (it == 1) eval[j] = eval[j] || !in_bits(E.clean, u[j]);
    }
    // most members stay and have nothing to settle
    if (!__any_sync(0xffffffffu, u[j] >= 0 && (oc != O_STAY || eval[j]))) continue;
    const bool need = u[j] >= 0 && oc == O_NONE;
    if (__any_sync(0xffffffffu, need)) {
      int c = cu[j];
      if (V == DC_HB && need) c = (int)(*flag_word<V>(E, u[j]) & (unsigned)kColorMask);
      const int r = find_witness<V>(need, u[j], c, i, inl);
      if (need) oc = r;
    }
    settle<V>(T, it, ring, oc, u[j], i, eval[j], need && oc == O_NONE);
  }
}

// MARK: PUSH and PULL side by side (the member search does not need the
// marks; HI's first iteration pushes first, because its members have no
// witnesses yet and all of them push).
template <int V>
__device__ __noinline__ void phase_mark(Target T, int it, int ring, unsigned* ctr) {
  constexpr unsigned W = V == DC_HB ? 4 : 2;
  const Env& E = env();
  const LoopState& in = inputs();
  const Work& w = shared().work;
  Grabber gb(ctr, w, team_warp(), E.nwarps);
  unsigned i;
#pragma unroll 1
  while (gb.next(i)) {
    if (i < w.units) {
      push_unit<V>(T, E.qb[0].units[i >> w.us], E.qb[0].gmask, (int)(i & ((1u << w.us) - 1)), 1 << w.us);
    } else if (i < w.members) {
      // Entries of a long row searched inline; the rest goes on beside the
      // next phase's mexes, a piece per warp.  Each 128 are a chain of three
      // dependent loads, and HI's searches mostly go on to the end of the
      // row: none inline took R-MAT scale 24 from 85.5 to 81.4 ms a batch and
      // scale 16 from 3.37 to 2.92 against 512 for a member that has its warp
      // alone and 128 else.  HB's end early (2 in 3 within 128; none inline
      // is 2 % slower at scale 16).
      pull_members<V, W>(T, it, ring, (i - w.units) << w.ms, 1u << w.ms,
                         (unsigned)min((long long)in.m_len[ring], E.mem_cap), V == DC_HI ? 0 : 128);
    } else {
      push_batchA<V>(T, E.qb[0].itemsA, (unsigned)min((long long)in.q[Q_PUSH].countA, E.qb[0].capA),
                     batch_item(i - w.members, w.as));
    }
  }
  finish_push(T);
}

// SCAN over one piece of a unit: nothing to look for once another piece of
// the row has a hit; the row's last piece settles the member.
template <int V>
__device__ __noinline__ void scan_piece(Target T, int it, int ring, int4 un, unsigned* gm, int sub, int ps) {
  const Env& E = env();
  const int u = un.x;
  const uint4 head = ld_cg(reinterpret_cast<const uint4*>(gm));
  const Span sp = span_of<V>(E, u);
  const int cu = (int)(*flag_word<V>(E, u) & (unsigned)kColorMask);
  const int pu = V == DC_HB ? E.g.prop[u] : 0;
  const int size = kScanUnit >> ps;
  const int s_lo = (int)head.w + un.y * kScanUnit + sub * size, s_hi = min(sp.len, s_lo + size);
  if (head.y == 0u && scan_span<V>(sp.at, s_lo, s_hi, u, cu, pu, sp.prior) && lane_id() == 0) atomicExch(&gm[1], 1u);
  __threadfence();
  __syncwarp();
  int last = 0;
  if (lane_id() == 0) last = atomicAdd(&gm[0], 1u) == (unsigned)(un.w << ps) - 1u;
  if (!__any_sync(0xffffffffu, last)) return;
  __threadfence();
  int oc = O_NONE;
  if (lane_id() == 0) oc = ld_cg(&gm[1]) != 0u ? O_STAY : O_LEAVE;
  settle<V>(T, it, ring, oc, u, head.z, false, false);
}

// SCAN and EVAL side by side.
template <int V>
__device__ __noinline__ void phase_eval(Target T, int it, int ring, unsigned* ctr, int mode, int* out) {
  const Env& E = env();
  const LoopState& in = inputs();
  const QueueBufs& sq = E.qb[1];
  const QueueBufs& eq = E.qb[2];
  const Work& w = shared().work;
  Grabber gb(ctr, w, team_warp(), E.nwarps);
  unsigned i;
#pragma unroll 1
  while (gb.next(i)) {
    if (i < w.units) {
      const int4 un = sq.units[i >> w.us];
      scan_piece<V>(T, it, ring, un, sq.gmask + un.z, (int)(i & ((1u << w.us) - 1)), w.us);
    } else if (i < w.members) {
      reduce_unit<V>(eq.units[i - w.units], eq.gmask, mode, true, out);
    } else {
      reduce_batchA<V>(eq.itemsA, (unsigned)min((long long)in.q[Q_EVAL + ring].countA, eq.capA),
                       batch_item(i - w.members, w.as), true, out);
    }
  }
}

// First colour change of v since the index was built (c0: its colour
// until then): queue v's row, in chunks, for the append phase.  An item is
// (v, chunk | bin << 21), bin = c0's count bin.  An overflowing queue turns
// the index off for the rest of the batch.
constexpr int kAppendChunk = 512;  // slots per append-phase item: 4 rounds of 4 loads per lane
constexpr int kChunkBits = 21;     // rows of up to 2^21 append chunks (2^30 slots)

__device__ __noinline__ void push_first(int v, int c0) {
  const Env& E = env();
  const int L = E.g.len[v];
  const int c = L > 0 ? (L + kAppendChunk - 1) / kAppendChunk : 0;
  if (c == 0) return;
  const unsigned b = atomicAdd(&E.ls->a_count, (unsigned)c);
  if ((long long)b + c > E.hri.cap_a) {
    atomicExch(&E.ls->hri_off, 1u);
    return;
  }
  const int bin = c0 < kHriBins - 1 ? c0 : kHriBins - 1;
#pragma unroll 1
  for (int q = 0; q < c; ++q) E.hri.alist[b + q] = make_int2(v, q | (bin << kChunkBits));
}

// Append phase: every vertex whose colour changed for the first time since
// the index was built joins the change list of each indexed neighbour, and
// leaves that neighbour's count of unchanged neighbours of its launch-start
// colour.
__device__ __noinline__ void phase_append(unsigned* ctr) {
  const Env& E = env();
  const HriBufs& H = E.hri;
  // an overflowed queue has unwritten items, and the index is off anyway
  if (inputs().hri_off != 0u) return;
  Grabber gb(ctr, (unsigned)min((long long)inputs().a_count, H.cap_a), team_warp(), E.nwarps);
  unsigned i;
#pragma unroll 1
  while (gb.next(i)) {
    const int2 it = H.alist[i];
    const int v = it.x;
    const int chunk = it.y & ((1 << kChunkBits) - 1);
    const int bin = it.y >> kChunkBits;
    const int L = E.g.len[v];
    const int* adj = E.g.adj + E.g.off[v];
    const int s_lo = chunk * kAppendChunk, s_hi = min(L, s_lo + kAppendChunk);
#pragma unroll 1
    for (int r0 = s_lo + lane_id(); r0 < s_hi; r0 += 128) {
      int uu[4], hh[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) uu[j] = r0 + j * 32 < s_hi ? adj[r0 + j * 32] : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) hh[j] = uu[j] >= 0 ? H.hid[uu[j]] : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (hh[j] < 0) continue;
        const int h = hh[j];
        const int slot = atomicAdd(&H.xcnt[h], 1);
        if ((long long)slot < H.xoff[h + 1] - H.xoff[h]) H.xv[H.xoff[h] + slot] = v;
        if (h < H.cap_hist && bin < kHriBins - 1) atomicSub(&H.hist[(long long)h * kHriBins + bin], 1);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------
// COMMIT and line phases
// ---------------------------------------------------------------------
// Item i of a queue: class A items first, then units with chunk 0.
__device__ __forceinline__ int queue_item(const QueueBufs& qb, unsigned cA, unsigned total, unsigned i) {
  if (i < cA) return qb.itemsA[i];
  if (i < total) {
    const int4 un = qb.units[i - cA];
    if (un.y == 0) return un.x;
  }
  return -1;
}

// COMMIT of the loop over the vertices whose state changes: the EVAL queue
// (new colour, clean), which holds every vertex that enters, and the leaving
// ones.  The vertices that push in the next iteration (new, changed, or --
// HI -- changed by the commit before) enter its PUSH queue.
template <int V>
__device__ __noinline__ void phase_commit(Target T, int it, int ring) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const GraphDev& g = E.g;
  const LoopState& in = inputs();
  const int* rows = E.qb[1].itemsA;
  const unsigned nq = in.ev_rows[ring];
  const unsigned total = nq + in.m_out[ring];
  int cmax_local = -1;
  long long ent = 0, ent_x = 0;  // live entries of the vertices that enter, of the indexed ones
#pragma unroll 1
  for (unsigned i = team_warp() * 32 + lane_id(); i < total; i += E.nwarps * 32) {
    const int v = i < nq ? rows[i] : E.mout[i - nq];
    unsigned* fw = flag_word<V>(E, v);
    const unsigned word = *fw;
    if (i >= nq) {
      *fw = word & ~kInF;
      clear_bit(E.inF, v);
      continue;
    }
    clear_bit(E.inE, v);
    if (E.wit[v] == kNoWitness) continue;  // its search failed
    const int pc = V == DC_HI ? g.prev[v] : 0;
    const int oc = (int)(word & (unsigned)kColorMask);
    const bool isnew = !(word & kInF);
    const int nc = E.ncolor[v];
    // a member changed by the commit before pushes once more: its previous
    // colour differs from the one it pushed with
    const bool again = V == DC_HI && !isnew && pc != oc;
    g.prev[v] = (V == DC_HB && isnew) ? (oc | kNewBit) : oc;
    *fw = (unsigned)nc | kInF;  // also clears the mark
    set_bit(E.clean, v);
    if (isnew) {
      set_bit(E.inF, v);
      const int lv = g.live[v];
      ent += lv;
      if (E.hri.min_live > 0 && lv >= E.hri.min_live) ent_x += lv;
    }
    if (nc != oc) {
      if (V == DC_HB) {
        g.color[v] = nc;
        if (E.hri_split) E.c8[v] = to_c8(nc);
        if (E.gchg) atomicAdd(&E.gchg[E.gid[v]], 1);
      } else if (E.hri_on && mark_bit(E.hri.bmF, v)) {
        push_first(v, oc);
      }
      cmax_local = max(cmax_local, nc);
    }
    if (isnew || again || nc != oc) stage(T, v);
  }
  __syncwarp();
  const int m = __reduce_max_sync(0xffffffffu, cmax_local);
  if (lane_id() == 0 && m >= 0) {
    atomicMax(&E.st->cmax, m);
    atomicExch(&E.ls->chg[ring], 1);
  }
  if (__any_sync(0xffffffffu, ent > 0)) {
    ent = warp_sum_ll(ent);
    ent_x = warp_sum_ll(ent_x);
    if (lane_id() == 0) {
      long long* c = sh.cov[warp_id()];
      c[0] -= 2ll * it * ent;
      c[1] += ent;
      c[2] -= 2ll * it * ent_x;
      c[3] += ent_x;
    }
  }
  finish_push(T);
}

// Rebuilds the member list from the membership bits, in vertex order within
// blocks of 1024 vertices: drops the entries of members that left, and
// gives a list that grew in push order its locality back.
__device__ __noinline__ void phase_rebuild() {
  const Env& E = env();
  const long long words = ((long long)E.g.n + 31) / 32;
#pragma unroll 1
  for (long long w0 = team_warp() * 32ll; w0 < words; w0 += E.nwarps * 32ll) {
    const long long w = w0 + lane_id();
    const unsigned bits = w < words ? E.inF[w] : 0u;
    const int c = __popc(bits);
    const int incl = warp_incl_scan(c);
    const int tot = __shfl_sync(0xffffffffu, incl, 31);
    if (tot == 0) continue;
    unsigned base = 0;
    if (lane_id() == 0) base = atomicAdd(&E.ls->m_build, (unsigned)tot);
    base = __shfl_sync(0xffffffffu, base, 0);
    unsigned todo = __ballot_sync(0xffffffffu, c > 0);
#pragma unroll 1
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const unsigned b = __shfl_sync(0xffffffffu, bits, l);
      const int ex = __shfl_sync(0xffffffffu, incl - c, l);
      if ((b >> lane_id()) & 1u) {
        const long long at = (long long)base + ex + __popc(b & lanemask_lt());
        if (at < E.mem_cap) E.mem[at] = (int)((w0 + l) * 32 + lane_id());
      }
    }
  }
}

enum Commit {
  C_SEED_DEL = 1, // HI deleteEdge: commit if changed, F0 += v, clear bmA
  C_SEED_INS = 2, // HI insEdge: commit always, F0 += v, clear bmC
  C_SEED_HB = 3,  // HB processChangeEdge: commit if changed, F0 += v, clear bmA
  C_CLEAR_A = 4   // clear bmA only
};

// COMMIT of the seeding: the vertices that change enter F0 (bmB, the loop's
// membership bits, keeps them distinct).
template <int V>
__device__ __noinline__ void phase_seed_commit(int buf, int q, int kind, int ch) {
  const Env& E = env();
  const GraphDev& g = E.g;
  const QueueBufs& qb = E.qb[buf];
  const QCount& qc = inputs().q[q];
  const unsigned cA = (unsigned)min((long long)qc.countA, qb.capA);
  const unsigned total = cA + (unsigned)min((long long)qc.countU, qb.capU);
  const Target T = {0, Q_PUSH, R_ROWS, ch};
  int items = 0;
  int cmax_local = -1;
#pragma unroll 1
  for (unsigned i = team_warp() * 32 + lane_id(); i < total; i += E.nwarps * 32) {
    const int v = queue_item(qb, cA, total, i);
    if (v < 0) continue;
    ++items;
    if (kind == C_SEED_INS)
      E.clean[v >> 5] = 0u;
    else
      E.bmA[v >> 5] = 0u;
    if (kind == C_CLEAR_A) continue;
    const int nc = E.ncolor[v];
    const int oc = g.color[v];
    if (nc == oc && kind != C_SEED_INS) continue;
    g.prev[v] = V == DC_HB ? (oc | kNewBit) : oc;
    g.color[v] = nc;
    if (V == DC_HB) *flag_word<V>(E, v) = (unsigned)nc;
    if (V == DC_HB && E.hri_split) E.c8[v] = to_c8(nc);
    // first colour change since the heavy-row index was built
    if (V == DC_HI && E.hri_on && nc != oc && mark_bit(E.hri.bmF, v)) push_first(v, oc);
    cmax_local = max(cmax_local, nc);
    if (mark_bit(E.inF, v)) {
      if (E.gf0) atomicAdd(&E.gf0[E.gid[v]], 1);
      stage(T, v);
    }
  }
  if (kind == C_CLEAR_A) return;
  __syncwarp();
  const int m = __reduce_max_sync(0xffffffffu, cmax_local);
  items = __reduce_add_sync(0xffffffffu, items);
  if (lane_id() == 0) {
    if (m >= 0) atomicMax(&E.st->cmax, m);
    if (items) atomicAdd(&E.st->seed_targets, (unsigned long long)items);
  }
  finish_push(T);
}

// F0 becomes the loop's first frontier: its vertices (whose bits are set in
// bmB, the membership bitmap) enter the member list without a witness.
template <int V>
__device__ __noinline__ void phase_frontier0() {
  const Env& E = env();
  LoopState* ls = E.ls;
  const QueueBufs& pq = E.qb[0];
  const QCount& pc = inputs().q[Q_PUSH];
  const unsigned cA = (unsigned)min((long long)pc.countA, pq.capA);
  const unsigned total = cA + (unsigned)min((long long)pc.countU, pq.capU);
#pragma unroll 1
  for (unsigned i0 = team_warp() * 32; i0 < total; i0 += E.nwarps * 32) {
    const int v = queue_item(pq, cA, total, i0 + lane_id());
    int lv = 0;
    if (v >= 0) {
      *flag_word<V>(E, v) |= kInF;
      E.wit[v] = -1;
      if (V == DC_HI && E.gcount) atomicAdd(&E.gcount[E.gid[v]], 1);
      lv = E.g.live[v];
    }
    const unsigned bal = __ballot_sync(0xffffffffu, v >= 0);
    if (!bal) continue;
    cover(lv, true, -1);  // covered by no frontier before the first
    // the list's tail, and the first iteration's length and member count
    unsigned base = 0;
    if (lane_id() < 3)
      base = atomicAdd(lane_id() == 0 ? &ls->m_tail : lane_id() == 1 ? &ls->m_len[1] : &ls->m_live[1],
                       (unsigned)__popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(bal & lanemask_lt());
    if (v >= 0) write_member(E, base, v);
  }
}

// Members of the next frontier once PULL (and SCAN) are through.
__device__ __forceinline__ long long next_members(const LoopState& in, int r) {
  return (long long)in.m_live[r] + (in.m_tail - in.m_len[r]) - in.m_out[r];
}

// The launch as a sequence of phases with a grid barrier after each.
enum Phase {
  P_D1, P_D2, P_D3, P_I1, P_I2, P_I3, P_I4, P_I5,  // HI seeding
  P_H1, P_H2, P_H3,                                // HB seeding
  P_F0, P_APPEND0,
  P_MARK, P_PULL, P_EVAL, P_COMMIT, P_APPEND, P_REBUILD, P_END
};

constexpr int kStateWords = sizeof(LoopState) / 4;

// The grid barrier, after which every CTA has a snapshot of the counters in
// shared memory (one round trip for all of them).  Phases and decisions read
// their inputs there; a counter that the phase under way changes may be
// newer or older in it and is not read.  `decide` then runs in thread 0 alone:
// the same few hundred instructions in 32 warps of every SM, cold in the
// instruction caches, were 2.6 us of each phase (R-MAT 24: 82.7 -> 76.7 ms a
// batch with this and the work of a phase planned here too, R-MAT 16 2.89 ->
// 2.68).
template <class F>
__device__ __forceinline__ bool sync_grid(DevState* st, unsigned long long timeout_ns, F decide) {
  Shared& sh = shared();
  __syncthreads();
  if (warp_id() == 0) {
    if (lane_id() == 0) sh.ok = barrier_wait(st, &st->ctl[1], sh.bar, timeout_ns) ? 1 : 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kStateWords; i += 32)
      if (i + lane_id() < kStateWords)
        reinterpret_cast<unsigned*>(&sh.snap)[i + lane_id()] =
            ld_cg(reinterpret_cast<unsigned*>(&st->ls) + i + lane_id());
    __syncwarp();
    if (lane_id() == 0) decide();
  }
  __syncthreads();
  return sh.ok != 0;
}
__device__ __noinline__ bool sync_grid(DevState* st, unsigned long long timeout_ns) {
  return sync_grid(st, timeout_ns, [] {});
}

// Phase timer: CTA 0 thread 0 reads %globaltimer after a barrier and charges
// the time since the last lap to the phase kind that just ended.
__device__ __forceinline__ void lap(int kind) {
  Shared& sh = shared();
  if (blockIdx.x != 0) return;
  const unsigned long long t = globaltimer_ns();
  sh.acc[kind] += t - sh.t_last;
  sh.t_last = t;
}

// The work items of MARK (it starts, push and pull: which halves) and EVAL.
template <int V>
__device__ __forceinline__ void plan_mark(int r, bool push, bool pull) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const LoopState& in = sh.snap;
  Work& w = sh.work;
  const unsigned cA = push ? (unsigned)min((long long)in.q[Q_PUSH].countA, E.qb[0].capA) : 0;
  const unsigned cU = push ? (unsigned)min((long long)in.q[Q_PUSH].countU, E.qb[0].capU) : 0;
  const unsigned len = pull ? (unsigned)min((long long)in.m_len[r], E.mem_cap) : 0;
  // units go in up to four pieces while there are warps for them; a short
  // member list is spread over the warps left
  w.us = unit_pieces(cU, E.nwarps);
  w.units = cU << w.us;
  const unsigned free = E.nwarps > 2 * w.units ? E.nwarps - w.units : E.nwarps / 2;
  w.ms = share(len, free, 5);
  if ((free << w.ms) < len) w.ms = V == DC_HB ? 7 : 6;  // as many as pull_members takes at once
  w.members = w.units + shares(len, w.ms);
  w.as = batch_share(cA, w.members, E.nwarps);
  w.total = w.members + shares(cA, w.as);
  w.sh = grab_share(w.total, E.nwarps);
}
__device__ __forceinline__ void plan_eval(int r) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const LoopState& in = sh.snap;
  Work& w = sh.work;
  const unsigned cS = (unsigned)min((long long)in.q[Q_SCAN].countU, E.qb[1].capU);
  const unsigned cA = (unsigned)min((long long)in.q[Q_EVAL + r].countA, E.qb[2].capA);
  const unsigned cU = (unsigned)min((long long)in.q[Q_EVAL + r].countU, E.qb[2].capU);
  w.us = unit_pieces(cS, E.nwarps);
  w.units = cS << w.us;
  w.members = w.units + cU;
  w.as = batch_share(cA, w.members, E.nwarps);
  w.total = w.members + shares(cA, w.as);
  w.sh = grab_share(w.total, E.nwarps);
}

// The phase after the one that just ended, and its work (one thread).
template <int V>
__device__ __noinline__ void next_phase(long long iter_cap) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const LoopState& in = sh.snap;
  Step& S = sh.step;
  const int r = S.r;
  int ph = S.ph;
  auto filled = [&](int q) { return in.q[q].countA + in.q[q].countU > 0; };
  bool next_it = false;
  switch (ph) {
    case P_D1: ph = filled(Q_S1) ? P_D2 : P_I1; break;
    case P_D2: ph = P_D3; break;
    case P_D3: ph = P_I1; break;
    case P_I1: ph = filled(Q_S2E) ? P_I2 : P_F0; break;
    case P_I2: ph = P_I3; break;
    case P_I3: ph = P_I4; break;
    case P_I4: ph = P_I5; break;
    case P_I5: ph = P_F0; break;
    case P_H1: ph = filled(Q_S1) ? P_H2 : P_F0; break;
    case P_H2: ph = P_H3; break;
    case P_H3: ph = P_F0; break;
    case P_F0: case P_APPEND0:
      if (ph == P_F0 && V == DC_HI && E.hri_on && in.a_count > 0) {
        ph = P_APPEND0;
        break;
      }
      lap(0);
      if (filled(Q_PUSH))
        next_it = true;
      else
        ph = P_END;
      break;
    case P_MARK:
      if (V == DC_HI && S.it == 1) {
        ph = P_PULL;
        break;
      }
      [[fallthrough]];
    case P_PULL:
      lap(1);
      if (in.ev_rows[r] + in.q[Q_SCAN].countU > 0) {
        ph = P_EVAL;
        break;
      }
      [[fallthrough]];
    case P_EVAL: {
      if (ph == P_EVAL) lap(2);
      const long long q = next_members(in, r);
      if (blockIdx.x == 0) sh.frontiers += q;
      if ((V == DC_HI && q == 0) || (V == DC_HB && in.ev_rows[r] == 0))
        ph = P_END;  // HB: every mex stands, no colour changes
      else
        ph = P_COMMIT;
      break;
    }
    case P_COMMIT: case P_APPEND:
      if (ph == P_COMMIT && V == DC_HB && in.chg[r] == 0) {
        lap(3);
        ph = P_END;
      } else if (ph == P_COMMIT && V == DC_HI && E.hri_on && in.a_count > 0) {
        ph = P_APPEND;
      } else {
        // the next iteration, with a rebuilt member list
        next_it = true;
      }
      break;
    case P_REBUILD:
      ph = P_MARK;
      lap(3);
      break;
    default: break;
  }
  if (next_it) {
    if (S.it > 0) lap(3);
    if (S.it >= iter_cap) {
      if (blockIdx.x == 0) atomicOr(&E.st->status, ST_ITER);
      ph = P_END;
    } else {
      ++S.it;
      S.r = S.rn;
      S.rn = S.rn == 2 ? 0 : S.rn + 1;
      ph = S.it > 1 && in.m_rebuild[S.r] != 0u ? P_REBUILD : P_MARK;
    }
  }
  S.ph = ph;
  S.ps = S.ps == 2 ? 0 : S.ps + 1;
  if (ph == P_MARK || ph == P_PULL)
    plan_mark<V>(S.r, ph == P_MARK, ph == P_PULL || V == DC_HB || S.it > 1);
  else if (ph == P_EVAL)
    plan_eval(S.r);
}

// The line phases of the seeding.
template <int V>
__device__ __noinline__ void phase_lines(int ph, const dc_change* lines, long long K, unsigned char* lflag, int ch) {
  const Env& E = env();
  const int* color = E.g.color;
  const bool pair = V == DC_HB || ph == P_I1;
  const Target T = {(short)(ph == P_I3 ? 1 : 2), (short)(ph == P_I3 ? Q_S2T : ph == P_I1 ? Q_S2E : Q_S1),
                    ph == P_I1 ? R_SAT : R_MEX, ch};
  unsigned* bm = ph == P_I3 ? E.clean : E.bmA;
#pragma unroll 1
  for (long long i = team_warp() * 32ll + lane_id(); i < K; i += E.nwarps * 32ll) {
    int a = -1, b = -1;
    if (ph == P_D1 || ph == P_H1 || lflag[i]) {
      const dc_change c = lines[i];
      const int ca = color[c.node1], cb = color[c.node2];
      if (V == DC_HB) {
        // H1: endpoints of equal-colour insertions and of all deletions
        if (c.inst == 0 || (c.inst == 1 && ca == cb)) {
          a = c.node1;
          b = c.node2;
        }
      } else if (ph == P_D1) {
        // deletion targets (and remember which insertions had equal colours)
        if (c.inst == 0) a = ca > cb ? c.node1 : c.node2;
        lflag[i] = (c.inst == 1 && ca == cb) ? 1 : 0;
      } else if (ph == P_I1) {
        // insertions still monochromatic -> both endpoints
        if (ca == cb) {
          a = c.node1;
          b = c.node2;
          lflag[i] = 2;
        }
      } else if (lflag[i] == 2) {
        // I3: targets
        a = E.wit[c.node1] < E.wit[c.node2] ? c.node1 : c.node2;
      }
    }
    if (a >= 0 && mark_bit(bm, a)) stage(T, a);
    if (pair && b >= 0 && mark_bit(bm, b)) stage(T, b);
  }
  finish_push(T);
}

// The common arguments into shared memory (all threads call; the caller
// synchronises).
__device__ __forceinline__ void setup_env(const RecolorParams& p) {
  Shared& sh = shared();
  if (threadIdx.x == 0) {
    Env& E = sh.E;
    E.g = p.g;
    E.st = p.st;
    E.ls = &p.st->ls;
    E.nwarps = gridDim.x * kWarps;
    E.loop_units = min(p.unit_slots, kLoopUnit);
#pragma unroll 1
    for (int i = 0; i < 3; ++i) E.qb[i] = p.qb[i];
    E.bmA = p.bmA;
    E.ncolor = p.ncolor;
    E.cp = p.cp;
    E.c8 = p.c8;
    E.hri = p.hri;
    E.hri_on = E.hri_split = false;
    E.mem = p.mem;
    E.mem_cap = p.mem_cap;
    E.mout = p.mout;
    E.wit = p.sat;
    E.inF = p.bmB;
    E.clean = p.bmC;
    E.inE = p.bmA;
    E.gid = p.gid;
    E.gcount = E.gchg = E.gf0 = nullptr;
    E.gskip = nullptr;
    sh.ccnt = sh.mcnt = 0;
    sh.bar = 0;
#pragma unroll 1
    for (int i = 0; i < 4; ++i) sh.acc[i] = 0;
    sh.frontiers = sh.sorted = 0;
    sh.step = Step{P_END, 0, 0, 1, 0};
  }
  if (lane_id() == 0) sh.scanned[warp_id()] = sh.idx_cov[warp_id()] = sh.idx_reads[warp_id()] = 0;
  if (lane_id() < 4) sh.cov[warp_id()][lane_id()] = 0;
}

}  // namespace

// One instantiation per variant, so each gets its own register allocation
// and no per-entry variant branches.
template <int V>
__global__ void __launch_bounds__(kThreads, 2) recolor_kernel(const __grid_constant__ RecolorParams p) {
  Shared& sh = shared();
  Env& E = sh.E;
  DevState* st = p.st;
  const long long gthreads = (long long)gridDim.x * blockDim.x;
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  // The structural launch failed (invalid line, pool exhausted, ...): the
  // batch is not applied.  Uniform: nothing writes pre_status here.
  if (ld_cg(&st->pre_status) != 0u) return;
  setup_env(p);
  if (threadIdx.x == 0) {
    E.hri_on = V == DC_HI && p.hri.min_live > 0;
    E.hri_split = V == DC_HB && p.hri.min_live > 0;
    sh.step.ph = V == DC_HI ? P_D1 : P_H1;
    if (p.gid) {
      E.gcount = V == DC_HI ? p.gcnt : nullptr;
      E.gf0 = p.gf0;
    }
  }
  // the counters the launch starts from
  if (threadIdx.x < kStateWords)
    reinterpret_cast<unsigned*>(&sh.snap)[threadIdx.x] =
        ld_cg(reinterpret_cast<unsigned*>(&st->ls) + threadIdx.x);
  __syncthreads();

  if (leader) st->t_recolor[0] = sh.t_last = globaltimer_ns();
  const long long K = p.k_dev ? *p.k_dev : p.k;
  constexpr int rmode = V == DC_HI ? M_MEX_ALL : M_MEX_PRIOR;

  while (true) {
    const int ph = sh.step.ph, r = sh.step.r, rn = sh.step.rn;
    const long long it = sh.step.it;
    if (ph == P_END) break;
    LoopState* ls = &st->ls;
    const LoopState& in = sh.snap;
    int* gprv = nullptr;  // HB, batched: colour changes per graph in the previous iteration
    if (V == DC_HB && E.gid) {
      gprv = p.gcnt + (it & 1 ? 0 : (long long)p.ngraphs);
      if (threadIdx.x == 0) {
        E.gchg = p.gcnt + (it & 1 ? (long long)p.ngraphs : 0);
        E.gskip = it > 1 ? gprv : nullptr;
      }
      __syncthreads();
    }
    // Counter the warps take work items from; the next phase's, last used two
    // phases ago, is cleared.
    const int ps = sh.step.ps;
    unsigned* ctr = &st->ctl[1].wctr[ps];
    if (leader) st->ctl[1].wctr[ps == 2 ? 0 : ps + 1] = 0u;
    // Unit size of the rows pushed for a seeding phase of about `items` work
    // items.
    auto units_for = [&](unsigned items) { return unit_slots_for(items, E.nwarps, p.unit_slots); };
    const int loop_units = E.loop_units;

    // ---------------- the phase ----------------
    switch (ph) {
      case P_H1:
        // packed (degree property, colour) words for this launch's gathers;
        // this phase's barrier publishes them
#pragma unroll 1
        for (long long v = gtid; v < p.g.n; v += gthreads) {
          const int c = p.g.color[v] & kColorMask;
          p.cp[v] = ((unsigned long long)(unsigned)p.g.prop[v] << 32) | (unsigned)c;
          if (E.hri_split) p.c8[v] = to_c8(c);
        }
        phase_lines<V>(ph, p.ch, K, p.lflag, units_for((unsigned)(K / 16)));
        break;
      case P_D1: case P_I1: case P_I3:
        phase_lines<V>(ph, p.ch, K, p.lflag, units_for((unsigned)(K / 16)));
        if (ph == P_I3) phase_seed_commit<V>(2, Q_S2E, C_CLEAR_A, 0);  // release the endpoint set
        break;
      case P_D2: case P_I2: case P_I4: case P_H2:
        // mex (or saturation size) of a queue's rows
        phase_reduce<V>(ph == P_I4 ? 1 : 2, ph == P_I2 ? Q_S2E : ph == P_I4 ? Q_S2T : Q_S1, ctr,
                        V == DC_HI && ph == P_I2 ? M_DISTINCT : rmode, false, ph == P_I2 ? p.sat : p.ncolor);
        break;
      case P_D3: case P_H3: case P_I5: {
        const int q = ph == P_I5 ? Q_S2T : Q_S1;
        phase_seed_commit<V>(ph == P_I5 ? 1 : 2, q, ph == P_I5 ? C_SEED_INS : ph == P_D3 ? C_SEED_DEL : C_SEED_HB,
                             units_for(in.q[q].countU + in.q[q].countA / 32));
        break;
      }
      case P_F0:
        // F0 is complete: it becomes the loop's first frontier, and all of
        // it pushes in the first iteration
        phase_frontier0<V>();
        if (E.gid) {
          // a graph whose seeding recoloured nothing never enters the loop
#pragma unroll 1
          for (long long gg = gtid; gg < p.ngraphs; gg += gthreads) p.gstate[gg] = p.gf0[gg] > 0 ? 1 : 2;
        }
        break;
      case P_APPEND0: case P_APPEND:
        // rows of vertices whose colour changed for the first time join
        // their indexed neighbours' change lists before these are read again
        phase_append(ctr);
        break;
      case P_MARK: case P_PULL:
        if (leader && ph == P_MARK) {
          // counters of the next iteration, last read two iterations ago, and
          // what the last one's APPEND and rebuild consumed
          ls->q[Q_EVAL + rn] = QCount{0, 0, 0, 0};
          ls->ev_rows[rn] = 0;
          ls->m_out[rn] = 0;
          ls->chg[rn] = 0;
          ls->a_count = 0;
          ls->m_build = 0;
        }
        if (V == DC_HB && E.gid && it > 1) {
          // graphs with no colour change in the previous iteration are done
          // (the reference's loop would have ended for them)
          for (long long gg = gtid; gg < p.ngraphs; gg += gthreads)
            if (p.gstate[gg] == 1 && gprv[gg] == 0) {
              p.gstate[gg] = 2;
              p.giters[gg] = (int)(it - 1);
            }
        }
        phase_mark<V>(Target{2, (short)(Q_EVAL + r), R_EVAL, loop_units, it == 1}, (int)it, r, ctr);
        break;
      case P_EVAL:
        if (leader) ls->q[Q_PUSH] = QCount{0, 0, 0, 0};  // consumed
        phase_eval<V>(Target{2, (short)(Q_EVAL + r), R_EVAL, loop_units, false}, (int)it, r, ctr, rmode, E.ncolor);
        break;
      case P_COMMIT: {
        const long long tail = (long long)in.m_tail;
        const long long q = next_members(in, r);
        if (leader) {
          // consumed; without EVAL rows nothing is pushed now
          if (in.ev_rows[r] == 0) ls->q[Q_PUSH] = QCount{0, 0, 0, 0};
          ls->q[Q_SCAN] = QCount{0, 0, 0, 0};
          ls->m_len[rn] = (unsigned)tail;
          ls->m_live[rn] = (unsigned)q;
          // entries of members that left, and entries appended since the list
          // was in vertex order
          const bool rebuild = (tail - q) + (tail - sh.sorted) > q / 2 + kMemSlack;
          ls->m_rebuild[rn] = rebuild ? 1u : 0u;
          if (rebuild) sh.sorted = q;
        }
        if (E.gid) {
#pragma unroll 1
          for (long long gg = gtid; gg < p.ngraphs; gg += gthreads) {
            if (V == DC_HB) {
              gprv[gg] = 0;  // the next iteration's counters
            } else if (p.gstate[gg] == 1 && ld_cg(&p.gcnt[gg]) == 0) {
              // a running graph whose next frontier is empty is done
              p.gstate[gg] = 2;
              p.giters[gg] = (int)it;
            }
          }
        }
        phase_commit<V>(Target{0, Q_PUSH, R_PUSH, loop_units}, (int)it, r);
        break;
      }
      case P_REBUILD:
        if (leader) ls->m_tail = ls->m_len[r] = in.m_live[r];
        phase_rebuild();
        break;
      default:
        break;
    }

    // ---------------- its barrier, and the next phase ----------------
    if (!sync_grid(st, p.bar_timeout_ns, [&] { next_phase<V>(p.iter_cap); })) return;
  }

  const long long it = sh.step.it;
  // ---------------- the end ----------------
  // the membership bits and the flags they stand for, and the clean bits
  {
    unsigned* inF = p.bmB;
    unsigned* clean = p.bmC;
    unsigned* inE = p.bmA;
    const long long words = ((long long)p.g.n + 31) / 32 + 1;
#pragma unroll 1
    for (long long w = gtid; w < words; w += gthreads) {
      unsigned bits = inF[w];
      if (bits) inF[w] = 0u;
      if (clean[w]) clean[w] = 0u;
      if (inE[w]) inE[w] = 0u;  // members that left with a mex queued
      if (V == DC_HI)
        for (; bits; bits &= bits - 1) {
          const long long v = w * 32 + __ffs(bits) - 1;
          p.g.color[v] &= kColorMask;
        }
    }
  }
  if (p.gid) {
    // graphs still running stop with the union's last iteration
#pragma unroll 1
    for (long long gg = gtid; gg < p.ngraphs; gg += gthreads)
      if (p.gstate[gg] == 1) p.giters[gg] = (int)it;
  }
  if (leader) {
    st->iterations = (unsigned long long)it;
    st->t_recolor[1] = globaltimer_ns();
#pragma unroll 1
    for (int i = 0; i < 4; ++i) st->phase_ns[i] = sh.acc[i];
    st->frontier_total = (unsigned long long)sh.frontiers;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long sn = 0, rd = 0;
#pragma unroll 1
    for (int w = 0; w < kWarps; ++w) {
      const long long* c = sh.cov[w];
      const long long all = sh.scanned[w] + c[0] + (2 * it + 1) * c[1];
      sn += all;
      // rows without an index count in full
      rd += all - sh.idx_cov[w] - c[2] - (2 * it + 1) * c[3] + sh.idx_reads[w];
    }
    if (sn) atomicAdd(&st->slots_scanned, (unsigned long long)sn);
    if (rd) atomicAdd(&st->slots_read, (unsigned long long)rd);
  }
}

// ---------------------------------------------------------------------
// Initial colouring: greedy lowest free colour in a priority order, as a
// Jones-Plassmann schedule (no reference counterpart: the reference takes
// its initial colours from an external tool, MG/README.txt:19-22).
//
// A vertex is coloured once every neighbour before it in the order is
// coloured, with the smallest colour none of those neighbours has.  Its
// neighbours after it are then exactly the uncoloured ones, so every vertex
// gets the colour the sequential greedy pass in that order gives it; the
// rounds only run the independent vertices of the order side by side.
// Order: larger g.prop first, ties by lower id (isPrior_RelativeOrdering's
// comparison); with g.prop all zero it is the vertex-id order.
//   P   pred[v] = neighbours before v         (all vertices, in units)
//   F   frontier F0 = vertices with pred 0
//   round (until the frontier is empty): one walk of each frontier row takes
//     the mex over the neighbours before v, which is v's colour, and one pred
//     from every neighbour after v; the ones that reach 0 form the next
//     frontier
// The vertices of a round are independent (an edge between two of them would
// leave the later one a pred), so a round reads no colour that it writes, and
// the next round starts behind its barrier.  A round of a few dozen vertices
// is bound by its chain of dependent trips to L2 and its barrier.  R-MAT scale
// 18, 3.8 M edges, LDF, 859 rounds: 18.0 ms; with a phase for the mex and one
// for the release, units of 4096 slots walked 32 at a time and a lane per
// class-A row it took 49.
// ---------------------------------------------------------------------
namespace {

// P over one unit, and a class-A batch: counts the neighbours of each row
// that come before it.
__device__ __noinline__ void pred_unit(int4 un, int* pred) {
  const GraphDev& g = env().g;
  const int v = un.x;
  const int L = g.len[v];
  const int* adj = g.adj + g.off[v];
  const int us = unit_span(L, un.w);
  const int s_lo = un.y * us, s_hi = min(L, s_lo + us);
  const int pv = g.prop[v];
  int cnt = 0;
#pragma unroll 1
  for (int s0 = s_lo + lane_id(); s0 < s_hi; s0 += 128) {
    int uu[4], pp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) uu[j] = s0 + j * 32 < s_hi ? adj[s0 + j * 32] : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) pp[j] = uu[j] >= 0 ? g.prop[uu[j]] : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) cnt += uu[j] >= 0 && is_prior(pp[j], uu[j], pv, v);
  }
  __syncwarp();
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane_id() == 0 && cnt) atomicAdd(&pred[v], cnt);
}

__device__ __noinline__ void pred_batchA(const int* items, unsigned cA, unsigned idx, int* pred) {
  Shared& sh = shared();
  const GraphDev& g = sh.E.g;
  const bool valid = idx < cA;
  const int v = valid ? items[idx] : 0;
  Rows& R = sh.rows[warp_id()];
  R.a[lane_id()] = v;
  R.b[lane_id()] = valid ? g.prop[v] : 0;
  R.c[lane_id()] = 0;
  const int T = number_rows(R, g.adj + (valid ? g.off[v] : 0), valid ? g.len[v] : 0);
#pragma unroll 1
  for (int s0 = lane_id(); s0 < T; s0 += 128) {
    int jj[4], uu[4], pp[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * 32;
      jj[r] = row_of(R, s);
      uu[r] = s < T ? R.at[jj[r]][s - R.excl[jj[r]]] : -1;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) pp[r] = uu[r] >= 0 ? g.prop[uu[r]] : 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (uu[r] >= 0 && is_prior(pp[r], uu[r], R.b[jj[r]], R.a[jj[r]])) atomicAdd(&R.c[jj[r]], 1);
  }
  __syncwarp();
  if (valid) pred[v] = R.c[lane_id()];
  __syncwarp();
}

// v's colour into the colour word and the packed word.
__device__ __forceinline__ void commit_init(const Env& E, int v, int c) {
  E.g.color[v] = c;
  *flag_word<DC_HB>(E, v) = (unsigned)c;
}

// U neighbours per lane: those after their row lose one pred; the ones that
// reach 0 are ready.
template <int U>
__device__ __forceinline__ void release(Target T, const int* uu, unsigned after, int* pred) {
  int left[U];
#pragma unroll
  for (int j = 0; j < U; ++j) left[j] = (after >> j) & 1u ? atomicSub(&pred[uu[j]], 1) : 0;
#pragma unroll
  for (int j = 0; j < U; ++j)
    if (left[j] == 1) stage(T, uu[j]);
}

// A round's walk of one unit of a row.  Returns the row's colour where this
// unit finished it, else -1.
__device__ __noinline__ int color_unit(Target T, int4 un, const unsigned* gmask, int* pred) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const int v = un.x;
  const int L = E.g.len[v];
  const int* adj = E.g.adj + E.g.off[v];
  const int us = unit_span(L, un.w);
  const int s_lo = un.y * us, s_hi = min(L, s_lo + us);
  const int limit = min(L, kMaskBits), nw = mask_words(L, M_MEX_PRIOR);
  const int pv = E.g.prop[v];
  unsigned* sm = sh.mask[warp_id()];
#pragma unroll 1
  for (int k = lane_id(); k < nw; k += 32) sm[k] = 0;
  __syncwarp();
  unsigned long long lm = 0;  // colours < 64 seen by this lane
  // eight slots per lane per round: a round is a chain of three dependent
  // trips to L2, whatever its width
  constexpr int U = 8;
#pragma unroll 1
  for (int r0 = s_lo + lane_id(); r0 < s_hi; r0 += 32 * U) {
    int uu[U];
    unsigned long long xx[U];
    unsigned after = 0;
#pragma unroll
    for (int j = 0; j < U; ++j) uu[j] = r0 + j * 32 < s_hi ? adj[r0 + j * 32] : -1;
#pragma unroll
    for (int j = 0; j < U; ++j) xx[j] = uu[j] >= 0 ? E.cp[uu[j]] : 0ull;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (uu[j] < 0) continue;
      if (!is_prior((int)(xx[j] >> 32), uu[j], pv, v)) {
        after |= 1u << j;
        continue;
      }
      const int c = (int)(unsigned)xx[j];
      if (c < 64)
        lm |= 1ull << c;
      else if (c < limit)
        atomicOr(&sm[c >> 5], 1u << (c & 31));
    }
    release<U>(T, uu, after, pred);
  }
  __syncwarp();
  fold_low(sm, lm);
  if (un.w > 1 && !merge_masks(const_cast<unsigned*>(gmask) + un.z, sm, nw, un.w)) return -1;
  int r = first_zero(sm, nw);
  __syncwarp();
  if (r < 0) r = slow_mex(v, M_MEX_PRIOR, kMaskBits);
  if (lane_id() == 0) commit_init(E, v, r);
  __syncwarp();
  return r;
}

// The same of a class-A batch.  Returns each lane's row's colour (-1: none).
__device__ __noinline__ int color_batchA(Target T, const int* items, unsigned cA, unsigned idx, int* pred) {
  Shared& sh = shared();
  const Env& E = sh.E;
  const bool valid = idx < cA;
  const int v = valid ? items[idx] : 0;
  Rows& R = sh.rows[warp_id()];
  unsigned long long* m64 = reinterpret_cast<unsigned long long*>(sh.mask[warp_id()]);
  m64[lane_id()] = 0ull;
  R.a[lane_id()] = v;
  R.b[lane_id()] = valid ? E.g.prop[v] : 0;
  const int S = number_rows(R, E.g.adj + (valid ? E.g.off[v] : 0), valid ? E.g.len[v] : 0);
#pragma unroll 1
  for (int s0 = lane_id(); s0 < S; s0 += 128) {
    int jj[4], uu[4];
    unsigned long long xx[4];
    unsigned after = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * 32;
      jj[r] = row_of(R, s);
      uu[r] = s < S ? R.at[jj[r]][s - R.excl[jj[r]]] : -1;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) xx[r] = uu[r] >= 0 ? E.cp[uu[r]] : 0ull;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const bool before = uu[r] >= 0 && is_prior((int)(xx[r] >> 32), uu[r], R.b[jj[r]], R.a[jj[r]]);
      if (uu[r] >= 0 && !before) after |= 1u << r;
      const int c = (int)(unsigned)xx[r];
      // a class-A row has at most 32 neighbours: its colour is below 64
      if (before && c < 64) atomicOr(reinterpret_cast<unsigned*>(&m64[jj[r]]) + (c >> 5), 1u << (c & 31));
    }
    release<4>(T, uu, after, pred);
  }
  __syncwarp();
  const int c = valid ? __ffsll((long long)~m64[lane_id()]) - 1 : -1;
  if (valid) commit_init(E, v, c);
  __syncwarp();
  return c;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 2) init_color_kernel(const __grid_constant__ RecolorParams p) {
  Shared& sh = shared();
  const Env& E = sh.E;
  setup_env(p);
  __syncthreads();
  DevState* st = p.st;
  const GraphDev& g = p.g;
  int* pred = p.pred;
  const unsigned gwarp = team_warp(), nwarps = E.nwarps;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  const int CH = E.loop_units;
  int ps = 0;
  auto ctr = [&]() -> unsigned* {
    unsigned* c = &st->ctl[1].wctr[ps];
    ps = ps == 2 ? 0 : ps + 1;
    if (leader) st->ctl[1].wctr[ps] = 0u;
    return c;
  };
  if (leader) st->t_recolor[0] = globaltimer_ns();
  // every vertex into the all-rows queue; packed (priority, colour) words
  const Target all = {2, Q_S1, R_ROWS, CH}, first = {0, 0, R_MEX, CH};
#pragma unroll 1
  for (long long v = gwarp * 32ll + lane_id(); v < g.n; v += nwarps * 32ll) {
    pred[v] = 0;
    p.cp[v] = ((unsigned long long)(unsigned)g.prop[v] << 32);
    stage(all, (int)v);
  }
  finish_push(all);
  if (!sync_grid(st, p.bar_timeout_ns)) return;
  // P
  {
    const QueueBufs& qb = p.qb[2];
    const QCount& qc = sh.snap.q[Q_S1];
    const unsigned cA = (unsigned)min((long long)qc.countA, qb.capA);
    const unsigned cU = (unsigned)min((long long)qc.countU, qb.capU);
    const int as = batch_share(cA, cU, nwarps);
    Grabber gb(ctr(), cU + shares(cA, as), gwarp, nwarps);
    unsigned i;
#pragma unroll 1
    while (gb.next(i)) {
      if (i < cU)
        pred_unit(qb.units[i], pred);
      else
        pred_batchA(qb.itemsA, cA, batch_item(i - cU, as), pred);
    }
  }
  if (!sync_grid(st, p.bar_timeout_ns)) return;
  // F0
#pragma unroll 1
  for (long long v = gwarp * 32ll + lane_id(); v < g.n; v += nwarps * 32ll)
    if (pred[v] == 0) stage(first, (int)v);
  finish_push(first);
  if (!sync_grid(st, p.bar_timeout_ns)) return;
  // queue counter slots 0..2 in turn, buffers 0 and 1
  int fs = 0, fb = 0;
  long long it = 0;
  int cmax = -1;
#pragma unroll 1
  while (sh.snap.q[fs].countA + sh.snap.q[fs].countU > 0) {
    if (it >= p.iter_cap) {
      if (leader) atomicOr(&st->status, ST_ITER);
      break;
    }
    ++it;
    const int ns = fs == 2 ? 0 : fs + 1;
    const int nb = fb ^ 1;
    if (leader) st->ls.q[ns == 2 ? 0 : ns + 1] = QCount{0, 0, 0, 0};
    const QueueBufs& fq = p.qb[fb];
    const QCount& fc = sh.snap.q[fs];
    const unsigned cA = (unsigned)min((long long)fc.countA, fq.capA);
    const unsigned cU = (unsigned)min((long long)fc.countU, fq.capU);
    const Target T = {(short)nb, (short)ns, R_MEX, CH};
    const int as = batch_share(cA, cU, nwarps);
    Grabber gb(ctr(), cU + shares(cA, as), gwarp, nwarps);
    unsigned i;
#pragma unroll 1
    while (gb.next(i))
      cmax = max(cmax, i < cU ? color_unit(T, fq.units[i], fq.gmask, pred)
                              : color_batchA(T, fq.itemsA, cA, batch_item(i - cU, as), pred));
    finish_push(T);
    if (!sync_grid(st, p.bar_timeout_ns)) return;
    fs = ns;
    fb = nb;
  }
  const int m = __reduce_max_sync(0xffffffffu, cmax);
  if (lane_id() == 0 && m >= 0) atomicMax(&st->cmax, m);
  if (leader) {
    st->iterations = (unsigned long long)it;
    st->t_recolor[1] = globaltimer_ns();
  }
}

cudaError_t launch_init_color(const RecolorParams& p, int grid, cudaStream_t s) {
  RecolorParams q = p;
  void* args[] = {&q};
  return cudaLaunchCooperativeKernel((const void*)init_color_kernel, dim3(grid), dim3(kThreads), args, sizeof(Shared),
                                     s);
}

cudaError_t launch_recolor(const RecolorParams& p, int grid, cudaStream_t s) {
  RecolorParams q = p;
  void* args[] = {&q};
  const void* fn = p.variant == DC_HB ? (const void*)recolor_kernel<DC_HB> : (const void*)recolor_kernel<DC_HI>;
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kThreads), args, sizeof(Shared), s);
}

int recolor_kernel_occupancy() {
  static_assert(sizeof(Shared) <= 48 * 1024, "no opt-in for more shared memory");
  int a = 0, b = 0, c = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, recolor_kernel<DC_HI>, kThreads, sizeof(Shared)) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, recolor_kernel<DC_HB>, kThreads, sizeof(Shared)) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, init_color_kernel, kThreads, sizeof(Shared)) != cudaSuccess)
    return 0;
  const int ab = a < b ? a : b;
  return ab < c ? ab : c;
}

}  // namespace dc

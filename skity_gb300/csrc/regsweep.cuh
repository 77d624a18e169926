// The sweep of sweep.cuh with the active edges held in registers.
//
// Same per-step restatement of WalkEdges (src/render/sw/sw_raster.cc:546-677)
// as LaneSweep, split into two loops, on a warp each (or in turns on one):
//
//   the walk (RegWalk) advances the active list step by step and only logs,
//   per step, one record per coverage interval -- its two edges' x before
//   and after the step and their dy -- into a shared-memory buffer;
//
//   the emission (RegEmit), run on each buffer the walk has filled, turns the
//   logged intervals of several rows into spans: a lane per interval for the
//   set-up (blit_trapezoid_row), then a lane per span.
//
// Each loop is short (the sweep was bound by instruction fetch and latency
// when a step's coverage was made inside the step), and the emission's lanes
// are filled by the spans of many rows instead of one row's.
//
// The walk's state:
//   * list position p of the active list is slot p / 32 of lane p % 32: x,
//     dx, dy, lower_y and a packed word (winding, curve count and shift,
//     quad slot) in registers; the quad-piece state an edge needs when a
//     piece ends sits in shared memory at the edge's quad slot, so a reorder
//     does not move it;
//   * what depends on the list alone -- which edges open and close
//     intervals, the nearest end of a piece -- is kept from step to step and
//     recomputed only when the list or a piece changes;
//   * windings are +-1, so their prefix sums are population counts of two
//     ballots.
// A path whose active list would exceed M edges (the form's size) is not swept
// here (RegWalk returns 0) and goes to LaneSweep.
#pragma once
#include "kernels.cuh"
#include "sweep.cuh"

namespace skc {

// Interval records the walk logs before they are emitted: a step with at
// most M active edges logs at most M / 2 + 1.
SKC_HD constexpr int RegRecords(int M) { return M == 32 ? 64 : M; }

// The packed word of an active edge: winding (2 bits, +-1), a flag for the
// edges a step has just inserted, curve count, curve shift, quad slot.
SKC_HD int32_t MakeWc(int winding, int count, int shift, int slot) {
  return (winding & 3) | ((count & 0x7F) << 8) | ((shift & 0xFF) << 16) |
         (int32_t)((uint32_t)slot << 24);
}
constexpr int32_t kWcNew = 4;
SKC_HD int WcWinding(int32_t wc) { return 2 - (wc & 3); }  // 1 -> 1, 3 -> -1
SKC_HD int WcCount(int32_t wc) { return (wc >> 8) & 0x7F; }
SKC_HD int WcShift(int32_t wc) { return (wc >> 16) & 0xFF; }
SKC_HD int WcSlot(int32_t wc) { return (int)((uint32_t)wc >> 24); }

// The flags of a logged interval beside its row (high 16 bits) and the
// step's alpha (low 8 bits).
enum : uint32_t {
  kRecClose = 0x100,     // the right edge is too close to its successor (full steps),
                         // or a trailing interval's precomputed test
  kRecFirst = 0x200,     // the step's first interval
  kRecTrailing = 0x400,  // left open by a culled right edge: no test against its neighbours
  kRecReal = 0x800       // after the set-up: spans are direct, not accumulated
};

// The interval records of a form, side 0 the left edge, side 1 the right one:
// x before the step; x after it (left: after the quad-piece update too); dy.
// The emission overwrites them by its set-ups (ul/ur, ll/lr, lDY/rDY).
template <int M>
struct RegLogT {
  static constexpr int kRecords = RegRecords(M);
  int32_t xa[2][kRecords], xb[2][kRecords], dy[2][kRecords];
  uint32_t meta[kRecords];
};
// Edge state by new list position (reorder and insertion), and the sort's
// keys: x and list position.
template <int M>
struct RegListT {
  int32_t x[M], dx[M], dy[M], low[M], wc[M];
  int32_t kx[M], kp[M];
};
// Accumulator flush: the nonzero entries of the row's difference array, then
// the runs they start.
template <int M>
struct RegRunsT {
  static constexpr int kEvents = 2 * M;  // entries a flush gathers at a time
  int32_t pos[kEvents], val[kEvents];
  int32_t run[kEvents + 2], sat[kEvents + 2];
};

// Per-warp shared block of the register sweep for active lists of up to
// M edges.
template <int M_>
struct RegSharedT {
  static constexpr int M = M_;
  RegLogT<M> log[1];
  int32_t start[32];   // first span of each set-up of the records being emitted
  int32_t q[8][M];     // quad-piece state by quad slot (RegQuad)
  uint8_t free_slot[M];  // quad slots no edge holds
  union {
    RegListT<M> p;  // during a step
    RegRunsT<M> f;  // between steps
  } u;
  SKC_HD RegListT<M>& list() { return u.p; }
  SKC_HD RegRunsT<M>& runs() { return u.f; }
};
// The same for a pass swept by two warps, one walking and one emitting: the
// walk fills one log while the other one is emitted.
template <int M_>
struct RegPairT {
  static constexpr int M = M_;
  RegLogT<M> log[2];
  int32_t start[32];
  int32_t q[8][M];
  uint8_t free_slot[M];
  RegListT<M> p;
  RegRunsT<M> f;
  int32_t filled[4];  // records of each log (-1: the walk gave up); whether it is the last
  SKC_HD RegListT<M>& list() { return p; }
  SKC_HD RegRunsT<M>& runs() { return f; }
};
// Host and device must agree on these sizes (the host sizes the launch).
static_assert(sizeof(RegSharedT<32>) % 16 == 0, "RegSharedT keeps 16-byte alignment");
static_assert(sizeof(RegSharedT<64>) % 16 == 0, "RegSharedT keeps 16-byte alignment");
static_assert(sizeof(RegSharedT<128>) % 16 == 0, "RegSharedT keeps 16-byte alignment");
static_assert(sizeof(RegSharedT<256>) % 16 == 0, "RegSharedT keeps 16-byte alignment");
static_assert(sizeof(RegPairT<32>) % 16 == 0 && sizeof(RegPairT<64>) % 16 == 0 &&
                  sizeof(RegPairT<128>) % 16 == 0 && sizeof(RegPairT<256>) % 16 == 0,
              "RegPairT keeps 16-byte alignment");

SKC_HD long long LaneMax64(const Lanes& L, long long v) {
#ifdef SKC_WARP_LANES
  for (int o = 16; o > 0; o >>= 1) {
    long long t = __shfl_xor_sync(0xffffffffu, v, o);
    v = t > v ? t : v;
  }
#endif
  return v;
}
SKC_HD uint32_t LaneOr(const Lanes& L, uint32_t v) {
#ifdef SKC_WARP_LANES
  return __reduce_or_sync(0xffffffffu, v);
#else
  return v;
#endif
}
SKC_HD unsigned LeMask(const Lanes& L) { return (2u << L.lane) - 1u; }

// Quad-piece state of an edge at its quad slot: forward-difference position,
// steps and second differences, the last point (the shift is in the edge's
// packed word).
template <typename Sh>
SKC_HD void RegQuadPut(Sh& sh, int slot, const Edge& e) {
  sh.q[0][slot] = e.qx;
  sh.q[1][slot] = e.qy;
  sh.q[2][slot] = e.qdx;
  sh.q[3][slot] = e.qdy;
  sh.q[4][slot] = e.qddx;
  sh.q[5][slot] = e.qddy;
  sh.q[6][slot] = e.q_last_x;
  sh.q[7][slot] = e.q_last_y;
}
template <typename Sh>
SKC_HD void RegQuadGet(const Sh& sh, int slot, Edge* e) {
  e->qx = sh.q[0][slot];
  e->qy = sh.q[1][slot];
  e->qdx = sh.q[2][slot];
  e->qdy = sh.q[3][slot];
  e->qddx = sh.q[4][slot];
  e->qddy = sh.q[5][slot];
  e->q_last_x = sh.q[6][slot];
  e->q_last_y = sh.q[7][slot];
}

// v at the next list position (the last one's is undefined).
template <int S>
SKC_HD void LaneNext(const Lanes& L, const int32_t (&v)[S], int s, int32_t* out) {
#ifdef SKC_WARP_LANES
  int32_t t = __shfl_down_sync(0xffffffffu, v[s], 1);
  if (S > 1) {
    const int32_t u = __shfl_sync(0xffffffffu, v[s + 1 < S ? s + 1 : s], 0);
    if (L.lane == 31) t = u;
  }
  *out = t;
#else
  *out = v[s + 1 < S ? s + 1 : s];
#endif
}
// v at the list position before (position 0: undefined).
template <int S>
SKC_HD void LanePrevOf(const Lanes& L, const int32_t (&v)[S], int s, int32_t* out) {
#ifdef SKC_WARP_LANES
  int32_t t = __shfl_up_sync(0xffffffffu, v[s], 1);
  if (S > 1) {
    const int32_t u = __shfl_sync(0xffffffffu, v[s > 0 ? s - 1 : 0], 31);
    if (L.lane == 0) t = u;
  }
  *out = t;
#else
  *out = v[s > 0 ? s - 1 : 0];
#endif
}

// Row accumulator of the sweep: the difference array, entries 0 .. width, and
// which of its up to 32 blocks of 1 << shift entries have been added to.  Few
// entries of a wide row are (two a span): with the range of the touched ones
// read from end to end, half the reads of 1,000-pixel paths of 64 verbs found
// nothing, three of four of 2,000-pixel ones (20,000 paths on 2048 x 2048
// 157 -> 152 ms, long strokes 8.2 -> 7.8, narrow paths as before).
struct AccState {
  int32_t* diff;
  int left, width;
  int shift;
  int y;             // row being accumulated (kNaN32: none)
  uint32_t touched;  // a bit per block (this lane's adds)
  // a flush under way: blocks to read, entries read of the first of them, the
  // sum and its saturated value before it, the run open there
  bool flushing;
  int at;
  int32_t sum, sat;
  int open;    // entry the open run starts at (-1: none), its value is `sat`
};

SKC_HD void AccFlushBegin(const Lanes& L, AccState& a) {
  a.touched = LaneOr(L, a.touched);
  a.at = 0;
  a.sum = a.sat = 0;
  a.open = -1;
  a.flushing = true;
}

// The next runs of an accumulated row (SpanBuilder::Flush, sw_raster.cc:
// 103-136): the row's alphas are the saturated prefix sums of the difference
// array, and a run starts at every entry whose alpha differs from its left
// neighbour's.  Gathers the next nonzero entries (each is reset to zero) and
// leaves the runs they complete in f.run / sat, each ending where the
// next one starts; returns their number.  A run still open waits in `a` for
// the next call; the last one has alpha 0 (a span's two entries cancel).
template <int M>
SKC_HD int AccRuns(const Lanes& L, AccState& a, RegRunsT<M>& f) {
  constexpr int NL = Lanes::n;
  int ne = 0;
#pragma unroll 1
  while (a.touched && ne + NL <= RegRunsT<M>::kEvents) {
    const int i = ((Lanes::ffs(a.touched) - 1) << a.shift) + a.at + L.lane;
    const int32_t d = i <= a.width ? a.diff[i] : 0;
    const unsigned mask = L.ballot(d != 0);
    if (mask) {
      if (d != 0) {
        const int e = ne + Lanes::popc(mask & L.lt_mask());
        f.pos[e] = i;
        f.val[e] = d;
        a.diff[i] = 0;
      }
      ne += Lanes::popc(mask);
    }
    a.at += NL;
    if (a.at >> a.shift) {  // the block's end
      a.at = 0;
      a.touched &= a.touched - 1;
    }
  }
  int ns = 0;
  if (a.open >= 0) {
    if (L.leader()) {
      f.run[0] = a.open;
      f.sat[0] = a.sat;
    }
    ns = 1;
  }
  L.sync();
#pragma unroll 1
  for (int eb = 0; eb < ne; eb += NL) {
    const int e = eb + L.lane;
    const bool valid = e < ne;
    const int32_t incl = LaneScanIncl(L, valid ? f.val[e] : 0) + a.sum;
    const int32_t sat = min_(incl, 255);
    const int32_t before = LanePrev(L, sat, a.sat);
    const bool start = valid && sat != before;
    const unsigned starts = L.ballot(start);
    if (start) {
      const int r = ns + Lanes::popc(starts & L.lt_mask());
      f.run[r] = f.pos[e];
      f.sat[r] = sat;
    }
    ns += Lanes::popc(starts);
    a.sum = LaneBcast(L, incl, NL - 1);
    a.sat = LaneBcast(L, sat, NL - 1);
  }
  L.sync();
  if (!a.touched) {
    a.flushing = false;
    a.y = kNaN32;
  }
  if (ns > 0) {
    --ns;
    a.open = f.run[ns];
  }
  L.sync();
  return ns;
}

// Spans of the logged intervals [0, nrec), rows in order; `last`: and of the
// row still accumulated.  Chunks of one record per lane are set up at once;
// their spans are made in runs of rows that end with the first row that
// accumulates (an accumulated row's spans follow its direct ones in the pool,
// so the accumulator is flushed before a later row's spans are written).  One
// loop makes the spans of both kinds, a span per lane, so that the code that
// stores them is there once (the sweep's instruction fetch is its scarcest
// resource).
template <typename Sh, typename Sink>
SKC_HD void RegEmit(const Lanes& L, Sh& sh, RegLogT<Sh::M>& lg, Sink* sink, AccState& as, int nrec,
                    Fixed left_clip, Fixed right_clip, bool last) {
  constexpr int NL = Lanes::n;
  RegRunsT<Sh::M>& f = sh.runs();
  int32_t last_ur = 0, last_lr = 0;  // the previous chunk's last right edge
  // the chunk [lo, lo + nv): this lane's record's row, spans before it and
  // through it; the chunk's row starts and accumulating records
  int lo = 0, nv = 0, row = 0, excl = 0, incl = 0;
  bool spans = false;
  unsigned heads = 0, accs = 0;
  int a = 0;         // next record of the chunk
  int w = 0, g1 = 0;  // spans of the run under way
  int fi = 0, fn = 0, fy = 0;  // accumulated runs to store, their row
#pragma unroll 1
  for (;;) {
    bool kept = false;
    uint2 v = make_uint2(0, 0);
    int y = 0, x = 0, len = 0;
    uint8_t al = 0;
    if (fi < fn) {
      const int i = fi + L.lane;
      y = fy;
      if (i < fn) {
        const int x0 = f.run[i];
        x = as.left + x0;
        len = f.run[i + 1] - x0;
        al = (uint8_t)f.sat[i];
        kept = al != 0;
      }
      fi += NL;
    } else if (as.flushing) {
      fy = as.y;
      L.sync();
      fn = AccRuns(L, as, f);
      fi = 0;
      continue;
    } else if (w < g1) {
      // the set-up of span w + lane: set-ups are packed in span order, so
      // it is the number of set-ups that start at or before the span
      const uint32_t rel = (uint32_t)(excl - w);
      const uint32_t bits = LaneOr(L, (spans && rel < (uint32_t)NL) ? 1u << rel : 0u);
      const int before = Lanes::popc(L.ballot(spans && excl < w));
      const int g = w + L.lane;
      if (g < g1) {
        const int j = before + Lanes::popc(bits & LeMask(L)) - 1;
        const uint32_t mt = lg.meta[lo + j];
        TrapRow q;
        q.ul = lg.xa[0][lo + j];
        q.ur = lg.xa[1][lo + j];
        q.ll = lg.xb[0][lo + j];
        q.lr = lg.xb[1][lo + j];
        q.lDY = lg.dy[0][lo + j];
        q.rDY = lg.dy[1][lo + j];
        q.full = (uint8_t)(mt & 0xFF);
        q.real = (mt & kRecReal) != 0;
        y = (int)mt >> 16;
        TrapSpan(q, g - sh.start[j], x, len, al);
        kept = q.real;
        if (!kept) {
          int o0 = x - as.left, o1 = o0 + len;
          o0 = max_(o0, 0);
          o1 = min_(o1, as.width);
          if (o0 < o1) {
            if (al != 0) {
              as.touched |= (1u << (o0 >> as.shift)) | (1u << (o1 >> as.shift));
              AtomicAddI32(&as.diff[o0], (int32_t)al);
              AtomicAddI32(&as.diff[o1], -(int32_t)al);
            }
          }
        }
      }
      w += NL;
    } else if (a < nv) {
      // the run [a, b) of records: to the end of the first row that
      // accumulates
      const int row_a = LaneBcast(L, row, a);
      if (as.y != kNaN32 && as.y != row_a) {
        AccFlushBegin(L, as);
        continue;
      }
      int at = a;  // the record whose row ends the run
      if (as.y == kNaN32) {
        const unsigned m = accs & ~((1u << a) - 1u);
        at = m ? Lanes::ffs(m) - 1 : NL;
      }
      int b = nv;
      if (at < nv) {
        const unsigned h = heads & ~((2u << at) - 1u);
        if (h) b = Lanes::ffs(h) - 1;
        as.y = LaneBcast(L, row, at);
      }
      w = LaneBcast(L, excl, a);
      g1 = LaneBcast(L, incl, b - 1);
      a = b;
      continue;
    } else if (lo + nv < nrec) {
      // the next chunk's set-ups
      lo += nv;
      a = w = g1 = 0;
      const int i = lo + L.lane;
      const bool valid = i < nrec;
      nv = min_(NL, nrec - lo);
      TrapRow t;
      int32_t ul = 0, ur = 0, ll = 0, lr = 0;
      uint32_t meta = 0;
      t.lDY = t.rDY = 0;
      L.sync();
      if (valid) {
        ul = lg.xa[0][i];
        ll = lg.xb[0][i];
        t.lDY = lg.dy[0][i];
        ur = lg.xa[1][i];
        lr = lg.xb[1][i];
        t.rDY = lg.dy[1][i];
        meta = lg.meta[i];
      }
      const int32_t pur = LanePrev(L, ur, last_ur), plr = LanePrev(L, lr, last_lr);
      last_ur = LaneBcast(L, ur, NL - 1);
      last_lr = LaneBcast(L, lr, NL - 1);
      row = (int)meta >> 16;
      const uint8_t full = (uint8_t)(meta & 0xFF);
      const int prev_right = (meta & kRecFirst)
                                 ? FixedFloorToInt(left_clip)
                                 : FixedCeilToInt(max_(min_(right_clip, pur), plr));
      const Fixed cul = max_(ul, left_clip);
      bool nr = (meta & kRecClose) != 0;
      if (!(meta & kRecTrailing))
        nr = nr || prev_right > FixedFloorToInt(cul) || prev_right > FixedFloorToInt(ll);
      int cnt = 0;
      bool real = false;
      if (valid && TrapPrepare(t, cul, min_(right_clip, ur), max_(left_clip, ll),
                               min_(right_clip, lr), t.lDY, t.rDY, full, nr)) {
        cnt = TrapCount(t);
        real = t.real;
      }
      incl = LaneScanIncl(L, cnt);
      excl = incl - cnt;
      spans = cnt > 0;
      const unsigned some = L.ballot(spans);
      L.sync();
      if (spans) {  // the set-ups that make spans, packed from `lo`
        const int j = Lanes::popc(some & L.lt_mask());
        lg.xa[0][lo + j] = t.ul;
        lg.xa[1][lo + j] = t.ur;
        lg.xb[0][lo + j] = t.ll;
        lg.xb[1][lo + j] = t.lr;
        lg.dy[0][lo + j] = t.lDY;
        lg.dy[1][lo + j] = t.rDY;
        lg.meta[lo + j] = (meta & 0xFFFF00FFu) | (real ? kRecReal : 0u);
        sh.start[j] = excl;
      }
      L.sync();
      const int prow = LanePrev(L, row, kNaN32);
      heads = L.ballot(valid && row != prow);
      accs = L.ballot(spans && !real);
      continue;
    } else if (last && as.y != kNaN32) {
      AccFlushBegin(L, as);
      continue;
    } else {
      break;
    }
    if (kept) {
      kept = sink->keep(x, y, len, al);
      v = sink->pack(x, len, al);
    }
    sink->put_rows(L, kept, v, y, (unsigned)len);
  }
  L.sync();
}

// Slot s (warp-uniform) of a per-slot register.
template <int S, typename T>
SKC_HD T SlotGet(const T (&v)[S], int s) {
  if (Lanes::n == 1) return v[s];
  T r = v[0];
#pragma unroll
  for (int i = 1; i < S; ++i)
    if (s == i) r = v[i];
  return r;
}
template <int S, typename T>
SKC_HD void SlotSet(T (&v)[S], int s, T x) {
  if (Lanes::n == 1) {
    v[s] = x;
    return;
  }
#pragma unroll
  for (int i = 0; i < S; ++i)
    if (s == i) v[i] = x;
}

// Stores an active list by list position for a reorder, then loads it back.
template <int M>
SKC_HD void RegStage(RegListT<M>& t, int r, int32_t x, int32_t dx, int32_t dy, int32_t low,
                     int32_t wc) {
  t.x[r] = x;
  t.dx[r] = dx;
  t.dy[r] = dy;
  t.low[r] = low;
  t.wc[r] = wc;
}

template <int M, int S>
SKC_HD void RegLoad(const Lanes& L, const RegListT<M>& t, int m, int32_t (&x)[S],
                    int32_t (&dx)[S], int32_t (&dy)[S], int32_t (&low)[S], int32_t (&wc)[S]) {
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int p = s * Lanes::n + L.lane;
    if (p < m) {
      x[s] = t.x[p];
      dx[s] = t.dx[p];
      dy[s] = t.dy[p];
      low[s] = t.low[p];
      wc[s] = t.wc[p];
    }
  }
}

// The interval left open by the last left edge of a step (its right edge was
// culled), logged behind the step's other intervals, with its too-close test
// against the left edge's predecessor after the reorder (its new predecessor
// if it survives, else the last processed survivor before it).
template <int M, int S>
SKC_HD void RegTrailing(const Lanes& L, RegLogT<M>& lg, const int32_t (&x)[S],
                        const int32_t (&dx)[S], const int32_t (&low)[S], const int (&off)[S],
                        Fixed next_y, int m, int nr, int nrec, uint32_t meta, Fixed left_clip) {
  constexpr int NL = Lanes::n;
  // the left edge: position, x, dx, whether it goes on
  int32_t mine = -1, xa = 0, dxa = 0, la = 0;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    if (off[s] == nr && s * NL + L.lane < m) {
      mine = s * NL + L.lane;
      xa = x[s];
      dxa = dx[s];
      la = low[s];
    }
  }
  const int a = LaneMax(L, mine);
  xa = LaneBcast(L, xa, NL == 32 ? a & 31 : 0);
  dxa = LaneBcast(L, dxa, NL == 32 ? a & 31 : 0);
  const bool a_surv = LaneBcast(L, la, NL == 32 ? a & 31 : 0) > next_y;
  long long key = 0;
  bool found = false;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int p = s * NL + L.lane;
    if (p < m && low[s] > next_y) {
      const int32_t xi = x[s];
      const bool cand = a_surv ? (p != a && (xi < xa || (xi == xa && p < a))) : p < a;
      if (cand) {
        const long long kk = ((long long)xi << 32) | (unsigned)p;
        if (!found || kk > key) key = kk;
        found = true;
      }
    }
  }
  const bool any = L.ballot(found) != 0;
  if (!found) key = (long long)kMinS32 << 32;
  key = LaneMax64(L, key);
  const int32_t pred_x = any ? (int32_t)(key >> 32) : left_clip;
  const bool tc = wadd(pred_x, kFixed1) >= wsub(xa, iabs_(dxa));
  if (L.leader()) {
    const int at = nrec + nr;
    lg.xa[1][at] = lg.xb[1][at] = kMaxS32;  // the right clip
    lg.dy[1][at] = 0;
    lg.meta[at] = meta | kRecTrailing | (nr == 0 ? kRecFirst : 0u) |
                  (((meta & 0xFF) == 0xFF && tc) ? kRecClose : 0u);
  }
}

// An edge moved left of an earlier one.  The reference ripples each such
// edge backwards (backward_insert_edge_based_on_x), which leaves the list
// stably sorted by new x; its crossing check then compares an edge with its
// predecessor at that moment: the latest (in sorted order) earlier-listed
// edge whose x is not greater.  Sorts the (x, list position) keys by odd-even
// transposition (the list is nearly sorted, so few phases run), finds each
// edge's predecessor by a short backward scan, reorders the list and returns
// whether this lane saw a crossing.
template <int M, int S>
SKC_HD bool RegSort(const Lanes& L, RegListT<M>& t, int m, int32_t (&x)[S], int32_t (&dx)[S],
                    int32_t (&dy)[S], int32_t (&low)[S], int32_t (&wc)[S]) {
  constexpr int NL = Lanes::n;
  int32_t* kx = t.kx;
  int32_t* kp = t.kp;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int p = s * NL + L.lane;
    if (p < m) {
      kx[p] = x[s];
      kp[p] = p;
      t.dx[p] = dx[s];
    }
  }
  L.sync();
  bool dirty_prev = true;
#pragma unroll 1
  for (int phase = 0; phase < m + 2; ++phase) {
    bool swapped = false;
#pragma unroll 1
    for (int i = 2 * L.lane + (phase & 1); i + 1 < m; i += 2 * NL) {
      const int32_t xa = kx[i], xb = kx[i + 1];
      const int32_t pa = kp[i], pb = kp[i + 1];
      if (xb < xa || (xb == xa && pb < pa)) {
        kx[i] = xb;
        kx[i + 1] = xa;
        kp[i] = pb;
        kp[i + 1] = pa;
        swapped = true;
      }
    }
    L.sync();
    const bool dirty = L.ballot(swapped) != 0;
    if (!dirty && !dirty_prev) break;
    dirty_prev = dirty;
  }
  bool cross = false;
#pragma unroll 1
  for (int r = L.lane; r < m; r += NL) {
    const int pr = kp[r];
    int q = r - 1;
#pragma unroll 1
    while (q >= 0 && kp[q] > pr) --q;
    if (q >= 0 && wadd(kx[q], t.dx[kp[q]]) > wadd(kx[r], t.dx[pr])) cross = true;
  }
  L.sync();
  // rank of each list position, by way of the wc row
#pragma unroll 1
  for (int r = L.lane; r < m; r += NL) t.wc[kp[r]] = r;
  L.sync();
  int rank[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int p = s * NL + L.lane;
    rank[s] = p < m ? t.wc[p] : 0;
  }
  L.sync();
#pragma unroll
  for (int s = 0; s < S; ++s)
    if (s * NL + L.lane < m) RegStage<M>(t, rank[s], x[s], dx[s], dy[s], low[s], wc[s]);
  L.sync();
  RegLoad<M, S>(L, t, m, x, dx, dy, low, wc);
  L.sync();
  return cross;
}

// WalkEdges over the pass's sorted edges W[0, n), logging the intervals of
// rows [row_lo, row_hi).  hand(records, last) takes a log that is full (or the
// last one) and returns the log to fill next.  Returns 0 if the active list
// would exceed M edges.
template <typename Sh, typename Hand>
SKC_HD int RegWalk(const Lanes& L, Sh& sh, const Edge* W, int n, bool even_odd, int row_lo,
                   int row_hi, int start_y, int stop_y, Fixed left_clip, Hand&& hand) {
  constexpr int NL = Lanes::n;
  constexpr int M = Sh::M;
  constexpr int S = M / NL;
  constexpr int R = RegLogT<M>::kRecords;
  constexpr unsigned kFull = NL == 32 ? 0xffffffffu : 1u;
  RegListT<M>& t = sh.list();
  RegLogT<M>* lg = &sh.log[0];
  const int winding_mask = even_odd ? 1 : -1;
  const Fixed y_stop = IntToFixed(stop_y);
  int32_t x[S], dx[S], dy[S], low[S], wc[S];
  int off[S];  // where the edge logs: side * R + its interval of the step; < 0: it does not

  Fixed y = max_(W[0].upper_y, IntToFixed(start_y));
  // initial activation: the edges with upper_y <= y, in their sorted order
  int k = 0;
#pragma unroll 1
  for (int base = 0; base < n; base += NL) {
    const int i = base + L.lane;
    const unsigned mask = L.ballot(i < n && W[i].upper_y <= y);
    k += Lanes::popc(mask);
    if (mask != kFull) break;
  }
  if (k > M) return 0;
  int m = k;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int p = s * NL + L.lane;
    x[s] = dx[s] = dy[s] = low[s] = wc[s] = 0;
    off[s] = -1;
    if (p < m) {
      Edge e = W[p];
      GoY(&e, y);
      x[s] = e.x;
      dx[s] = e.dx;
      dy[s] = e.dy;
      low[s] = e.lower_y;
      wc[s] = MakeWc(e.winding, e.curve_count, e.curve_shift, p);
      if (e.curve_count > 0) RegQuadPut(sh, p, e);
    }
    sh.free_slot[p] = (uint8_t)(M - 1 - p);  // taken from the end: slots m, m + 1, ...
  }
  int n_free = M - m;
  Fixed pend_y = k < n ? W[k].upper_y : kMaxS32;
  // of the list: intervals a step logs (and how many of them a right edge
  // closes), whether one stays open, the lowest end of a piece, the lowest
  // one past y
  int nr = 0, K = 0;
  bool final_in = false;
  Fixed lmin = kMaxS32, lnext = kMaxS32;
  bool cross = false, changed = true;
  // records to log before the hand-over: few at first, so that the emission of
  // a short pass does not wait for a full log (110,000 glyphs 6.99 -> 6.82 ms,
  // 64 canvases of fills 13.46 -> 13.39)
  int nrec = 0, limit = min_(R, 16);
  L.sync();

#pragma unroll 1
  for (;;) {
    bool done = false;
#pragma unroll 1
    for (;;) {
      if (changed) {
        // ---- what the list determines
        int32_t carry = 0;
        int nl = 0;
        nr = 0;
        int32_t l0 = kMaxS32, l1 = kMaxS32;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          if (s == 0 || s * NL < m) {
            const bool valid = s * NL + L.lane < m;
            const bool neg = (wc[s] & 2) != 0;
            const unsigned bp = L.ballot(valid && !neg), bn = L.ballot(valid && neg);
            const unsigned le = LeMask(L);
            const int32_t incl = carry + Lanes::popc(bp & le) - Lanes::popc(bn & le);
            const int32_t excl = incl - (neg ? -1 : 1);
            const bool in = (incl & winding_mask) != 0;
            const bool pin = (excl & winding_mask) != 0;
            const unsigned lm = L.ballot(valid && in && !pin), rm = L.ballot(valid && !in && pin);
            off[s] = -1;
            if (valid && in != pin)
              off[s] = in ? nl + Lanes::popc(lm & L.lt_mask())
                          : R + nr + Lanes::popc(rm & L.lt_mask());
            nl += Lanes::popc(lm);
            nr += Lanes::popc(rm);
            carry += Lanes::popc(bp) - Lanes::popc(bn);
            if (valid) {
              l0 = min_(l0, low[s]);
              if (low[s] > y) l1 = min_(l1, low[s]);
            }
          }
        }
        final_in = (carry & winding_mask) != 0;
        K = nr + (final_in ? 1 : 0);
        lmin = LaneMin(L, l0);
        lnext = LaneMin(L, l1);
        changed = false;
      }
      if (nrec + K > limit && nrec > 0) break;  // full: emit, then take the step
      Fixed nny = min_(lnext, pend_y);
      if (cross) nny = min_(nny, y + (kFixed1 >> kAccuracy));
      cross = false;
      if (m == 0) {  // nothing active: on to the next edge
        y = pend_y;
        if (y >= y_stop) {
          done = true;
          break;
        }
      } else {
        Fixed next_y = min_(nny, FixedCeilToFixed(y + 1));
        int y_shift = 0;
        if ((next_y - y) & (kFixed1 >> 2)) {
          y_shift = 2;
          next_y = y + (kFixed1 >> 2);
        } else if ((next_y - y) & (kFixed1 >> 1)) {
          y_shift = 1;
        }
        const uint8_t full = partial_alpha_h(0xFF, next_y - y);
        const int row = y >> 16;
        const bool log = K > 0 && row >= row_lo && row < row_hi;
        const uint32_t meta = ((uint32_t)row << 16) | full;

        // ---- A: advance every active edge, log the intervals
        int32_t xo[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          xo[s] = x[s];
          x[s] = wadd(x[s], dx[s] >> y_shift);  // GoYShift
        }
        if (log) {
#pragma unroll
          for (int s = 0; s < S; ++s) {
            if (s == 0 || s * NL < m) {
              uint32_t close = 0;
              if (full == 0xFF) {
                // edges_too_close(right edge, its successor before the step);
                // an edge still pending starts at next_y or later
                const int p = s * NL + L.lane;
                int32_t nxo = 0, ndx = 0;
                LaneNext<S>(L, xo, s, &nxo);
                LaneNext<S>(L, dx, s, &ndx);
                if (p + 1 < m && wadd(x[s], kFixed1) >= wsub(nxo, iabs_(ndx))) close = kRecClose;
              }
              if (off[s] >= 0) {
                const int at = off[s] + nrec;
                (&lg->xa[0][0])[at] = xo[s];
                (&lg->xb[0][0])[at] = x[s];
                (&lg->dy[0][0])[at] = dy[s];
                if (off[s] >= R) lg->meta[at - R] = meta | close | (off[s] == R ? kRecFirst : 0u);
              }
            }
          }
        }

        // ---- pieces that end in the step: the next quad piece, or the edge's end
        if (next_y >= lmin) {
          changed = true;
#pragma unroll 1
          for (int s = 0; s * NL < m; ++s) {  // one copy of the update for all slots
            const int32_t ls = SlotGet<S>(low, s), ws = SlotGet<S>(wc, s);
            if (s * NL + L.lane < m && ls <= next_y && WcCount(ws) > 0) {
              const int slot = WcSlot(ws);
              Edge e;
              RegQuadGet(sh, slot, &e);
              e.x = SlotGet<S>(x, s);
              e.y = next_y;
              e.dx = SlotGet<S>(dx, s);
              e.dy = SlotGet<S>(dy, s);
              e.lower_y = ls;
              e.winding = (int8_t)WcWinding(ws);
              e.curve_count = (int8_t)WcCount(ws);
              e.curve_shift = (uint8_t)WcShift(ws);
#pragma unroll 1
              while (e.lower_y <= next_y && e.curve_count > 0) {
                e.snapped_x = e.x;  // KeepContinuous (sw_edge.cc:294-297)
                e.snapped_y = e.y;
                if (!UpdateQuad(&e)) break;
              }
              RegQuadPut(sh, slot, e);
              SlotSet<S>(x, s, e.x);
              SlotSet<S>(dx, s, e.dx);
              SlotSet<S>(dy, s, e.dy);
              SlotSet<S>(low, s, e.lower_y);
              SlotSet<S>(wc, s, MakeWc(e.winding, e.curve_count, e.curve_shift, slot));
              const int o = SlotGet<S>(off, s);
              if (log && o >= 0 && o < R) (&lg->xb[0][0])[o + nrec] = e.x;
            }
          }
        }
        if (SKC_COLD(final_in && log))
          RegTrailing<M, S>(L, *lg, x, dx, low, off, next_y, m, nr, nrec, meta, left_clip);
        if (next_y >= lmin) {
          // ---- the edges that go on, in list order
          unsigned smask[S];
          int m2 = 0;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            smask[s] = L.ballot(s * NL + L.lane < m && low[s] > next_y);
            m2 += Lanes::popc(smask[s]);
          }
          if (m2 != m) {
            int r0 = 0, d0 = n_free;
#pragma unroll
            for (int s = 0; s < S; ++s) {
              if (s == 0 || s * NL < m) {
                const int p = s * NL + L.lane;
                const unsigned gone = L.ballot(p < m) & ~smask[s];
                if ((smask[s] >> (NL == 32 ? L.lane : 0)) & 1u)
                  RegStage<M>(t, r0 + Lanes::popc(smask[s] & L.lt_mask()), x[s], dx[s], dy[s],
                              low[s], wc[s]);
                else if (p < m)
                  sh.free_slot[d0 + Lanes::popc(gone & L.lt_mask())] = (uint8_t)WcSlot(wc[s]);
                r0 += Lanes::popc(smask[s]);
                d0 += Lanes::popc(gone);
              }
            }
            n_free = d0;
            m = m2;
            L.sync();
            RegLoad<M, S>(L, t, m, x, dx, dy, low, wc);
            L.sync();
          }
        }
        if (log) nrec += K;

        // ---- C: the list in stable order of the new x; intersections
        bool inv = false, crs = false;
        {
          int32_t sum[S];
#pragma unroll
          for (int s = 0; s < S; ++s) sum[s] = wadd(x[s], dx[s]);
#pragma unroll
          for (int s = 0; s < S; ++s) {
            if (s == 0 || s * NL < m) {
              const int p = s * NL + L.lane;
              int32_t px = 0, ps = 0;
              LanePrevOf<S>(L, x, s, &px);
              LanePrevOf<S>(L, sum, s, &ps);
              if (p > 0 && p < m) {
                inv = inv || px > x[s];
                crs = crs || ps > sum[s];
              }
            }
          }
        }
        if (L.ballot(inv || crs)) {
          if (L.ballot(inv)) {
            crs = RegSort<M, S>(L, t, m, x, dx, dy, low, wc);
            changed = true;
          }
          cross = L.ballot(crs) != 0;
        }
        y = next_y;
        if (y >= y_stop) {
          done = true;
          break;
        }
      }

      // ---- D: insert_new_edges (sw_raster.cc:207-247) as a merge
      if (pend_y <= y) {
        int c = 0;
#pragma unroll 1
        for (int base = k; base < n; base += NL) {
          const int i = base + L.lane;
          const unsigned mask = L.ballot(i < n && W[i].upper_y <= y);
          c += Lanes::popc(mask);
          if (mask != kFull) break;
        }
        if (SKC_COLD(m + c > M)) return 0;
        // the first new edge goes after every active edge with x <= its x,
        // each later one after the one before it and the active edges with
        // smaller x
        const int32_t x0 = W[k].x;
        int before[S];  // new edges before each active one
#pragma unroll
        for (int s = 0; s < S; ++s) before[s] = x[s] > x0 ? 1 : 0;
#pragma unroll 1
        for (int tb = 0; tb < c; tb += NL) {
          const int te = tb + L.lane;
          Edge e;
          int np = 0;
          if (te < c) e = W[k + te];
          const int32_t xt_mine = te < c ? e.x : 0;
          const int tn = min_(NL, c - tb);
#pragma unroll 1
          for (int j = 0; j < tn; ++j) {
            const int32_t xt = LaneBcast(L, xt_mine, j);
            const bool first = tb + j == 0;
            int cnt = 0;
#pragma unroll
            for (int s = 0; s < S; ++s) {
              if (s == 0 || s * NL < m) {
                const bool act = s * NL + L.lane < m;
                cnt += Lanes::popc(L.ballot(act && (x[s] <= x0 || (!first && x[s] < xt))));
                if (!first && x[s] > x0 && xt <= x[s]) before[s]++;
              }
            }
            if (j == L.lane || NL == 1) np = tb + j + cnt;
          }
          if (te < c) {
            const int slot = sh.free_slot[n_free - 1 - te];
            RegStage<M>(t, np, e.x, e.dx, e.dy, e.lower_y,
                           MakeWc(e.winding, e.curve_count, e.curve_shift, slot) | kWcNew);
            if (e.curve_count > 0) RegQuadPut(sh, slot, e);
          }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int p = s * NL + L.lane;
          if (p < m) RegStage<M>(t, p + before[s], x[s], dx[s], dy[s], low[s], wc[s]);
        }
        n_free -= c;
        m += c;
        k += c;
        pend_y = k < n ? W[k].upper_y : kMaxS32;
        L.sync();
        RegLoad<M, S>(L, t, m, x, dx, dy, low, wc);
        bool cross2 = false;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int p = s * NL + L.lane;
          if (p < m && (wc[s] & kWcNew)) {
            wc[s] &= ~kWcNew;
            if (p > 0 && wadd(t.x[p - 1], t.dx[p - 1]) > wadd(x[s], dx[s])) cross2 = true;
          }
        }
        L.sync();
        if (L.ballot(cross2)) cross = true;
        changed = true;
      }
    }
    lg = hand(nrec, done);
    limit = min_(R, 2 * limit);
    nrec = 0;
    if (done) break;
  }
  return 1;
}

}  // namespace skc

// Per-thread bodies of the raster kernels, host+device so the pipeline can
// also be executed on the CPU by tests (the GPU runs them through the
// __global__ wrappers in kernels.cu).
#pragma once
#include "kernels.cuh"
#include "edges.cuh"
#include "stroke.cuh"
#include "regsweep.cuh"

namespace skc {

// The whole geometry of a pass on one thread (the CPU execution of the
// pipeline; the GPU runs its two parts on a warp each, kernels.cu).
SKC_HDN void GeometryPass(const DevBatch& b, uint32_t p) {
  Lanes lanes;
  lanes.lane = 0;
  SortShared sh;
  StrokePass(b, p, lanes);
  EdgesPass(b, p, lanes, &sh);
}

// ---------------------------------------------------------------------------
// sweep: the span sink and the sweep passes
// ---------------------------------------------------------------------------
// SWSpanBrush::Brush clipping (sw_span_brush.cc:78-99); false = dropped
SKC_HD bool ClipSpan(int& x, int y, int& len, int W, int H) {
  if (y < 0 || y >= H) return false;
  if (x >= W || x + len < 0) return false;
  if (x < 0) {
    len += x;
    x = 0;
  }
  if (x + len >= W) len = W - x;
  return len > 0;
}

// keep() applies the clipping of SWSpanBrush::Brush and drops spans whose
// alpha & global alpha is 0 under src-over (they blend to nothing).  A raw
// sink (the passes of the path-clip stages) keeps every span of its rows as
// the raster made it, in the raw format of pack(); only sinks built with
// kRawCapable take that form (batches without path clips use the others).
template <bool kRawCapable>
struct SinkBase {
  int row0, row1, W, H;
  uint32_t ga;
  bool srcover;
  bool raw;
  SKC_HD bool keep(int& x, int y, int& len, uint8_t a) const {
    if (y < row0 || y >= row1) return false;
    if (kRawCapable && raw) return true;
    if (!ClipSpan(x, y, len, W, H)) return false;
    return !(srcover && (a & ga) == 0);
  }
  // A stored span: x | len << 16 and the alpha; raw: x (int32) and
  // len | alpha << 24.
  SKC_HD uint2 pack(int x, int len, uint32_t a) const {
    return (kRawCapable && raw) ? make_uint2((uint32_t)x, ((uint32_t)len & 0xFFFFFFu) | (a << 24))
                                : make_uint2((uint32_t)x | ((uint32_t)len << 16), a);
  }
};

SKC_HD unsigned long long LaneBcast64(const Lanes& L, unsigned long long v, int src) {
#ifdef SKC_WARP_LANES
  return __shfl_sync(0xffffffffu, v, src);
#else
  return v;
#endif
}

// Spans go to one device-wide pool handed out in chunks of `chunk` spans.
// A pass writes its rows one after another, each row contiguous -- a row
// that would run past the end of its chunk is moved to a fresh chunk -- and
// records (first span, count) per canvas row.  When the pool is exhausted
// the pass keeps taking chunks but writes nothing, so the allocator ends at
// the exact size the pass needs; the caller then sweeps again with a pool
// that large.  All members are warp-uniform; methods are called by the
// whole warp.
template <bool kRawCapable>
struct PoolSinkT : SinkBase<kRawCapable> {
  using SinkBase<kRawCapable>::keep;
  using SinkBase<kRawCapable>::pack;
  using SinkBase<kRawCapable>::row0;
  using SinkBase<kRawCapable>::row1;
  uint2* pool;
  uint64_t cap;                // pool capacity in spans
  unsigned long long* next;    // spans handed out so far
  uint32_t chunk;              // spans per chunk (holds any row of the pass)
  uint2* rows;                 // (first span, count) per row of [row0, row1)
  uint32_t* err;
  int cur_row;
  // positions in the pool (it has less than 2^32 spans; meaningless once dead)
  uint32_t row_start, cur, chunk_end;
  bool dead;
  uint32_t kept;
  unsigned long long frags;

  SKC_HD void finish_row(const Lanes& L) {
    if (!dead && cur > row_start && cur_row >= row0 && cur_row < row1 && L.leader())
      rows[cur_row - row0] = make_uint2(row_start, cur - row_start);
  }
  SKC_HD void row_begin(const Lanes& L, int y) {
    if (y == cur_row) return;
    finish_row(L);
    cur_row = y;
    row_start = cur;
  }
  // Room for `add` more spans after the `written` spans this step already
  // put at cur; returns cur (the row may have moved to a new chunk).
  SKC_HD uint32_t reserve(const Lanes& L, uint32_t written, uint32_t add) {
    if (SKC_LIKELY(written + add <= chunk_end - cur)) return cur;
    const uint32_t have = cur + written - row_start;
    if (have + add > chunk) {  // a row larger than a chunk (not expected)
      FlagError(err, 8);
      dead = true;
    }
    unsigned long long c = 0;
    if (L.leader()) {
#ifdef __CUDA_ARCH__
      c = atomicAdd(next, (unsigned long long)chunk);
#else
      c = *next;
      *next += chunk;
#endif
    }
    c = LaneBcast64(L, c, 0);
    if (c + chunk > cap) dead = true;
    if (!dead) {
      L.sync();
#pragma unroll 1
      for (uint32_t i = L.lane; i < have; i += Lanes::n) pool[c + i] = pool[row_start + i];
      L.sync();
    }
    cur = (uint32_t)c + (cur - row_start);
    row_start = (uint32_t)c;
    chunk_end = row_start + chunk;
    return cur;
  }
  SKC_HD uint2* span_ptr(uint32_t i) { return dead ? nullptr : pool + i; }
  // One span per lane (`kept`), rows in increasing order over the lanes, of
  // `len` pixels each: appended in lane order, every row that ends among them
  // entered in the row table, the last one left open.
  SKC_HD void put_rows(const Lanes& L, bool kept_, uint2 v, int y, unsigned len) {
    const unsigned km = L.ballot(kept_);
    if (!km) return;
    const uint32_t cnt = (uint32_t)Lanes::popc(km);
    const uint32_t at = reserve(L, 0, cnt);
    const unsigned below = km & L.lt_mask();
    const uint32_t mine = at + (uint32_t)Lanes::popc(below);
    if (kept_ && !dead) pool[mine] = v;
    const int py = LaneBcast(L, y, below ? 31 - clz_(below) : L.lane);
    const bool head = kept_ && (below ? py : cur_row) != y;
    const unsigned heads = L.ballot(head);
    if (heads) {
      const int last = 31 - clz_(heads);
      if (head && !dead) {
        // the first one ends the row left open, each but the last is a row
        if (L.lane == Lanes::ffs(heads) - 1 && mine > row_start && cur_row >= row0 &&
            cur_row < row1)
          rows[cur_row - row0] = make_uint2(row_start, mine - row_start);
        if (L.lane != last) {
          const unsigned next = heads & ~((2u << L.lane) - 1u);
          rows[y - row0] = make_uint2(
              mine, (uint32_t)Lanes::popc(km & ~L.lt_mask() & ((next & (0u - next)) - 1u)));
        }
      }
      cur_row = LaneBcast(L, y, last);
      row_start = at + (uint32_t)Lanes::popc(km & ((1u << last) - 1u));
    }
    commit(L, cnt, kept_ ? len : 0u);
  }
  // n: spans appended (warp-uniform); f: this lane's share of their
  // fragments (the shares are summed once, when the pass finishes)
  SKC_HD void commit(const Lanes&, uint32_t n, unsigned long long f) {
    cur += n;
    kept += n;
    frags += f;
  }
  // The accumulated spans of a row follow its direct spans (the reference
  // flushes a row's accumulator only after leaving the row,
  // SpanBuilder::Flush, sw_raster.cc:103-136): the runs of equal nonzero
  // saturated prefix sums of diff[lo, hi), in increasing x.  Returns false
  // when the row lies outside the canvas (diff not read).
  //
  // Each lane takes V consecutive entries per chunk of Lanes::n * V; a run
  // starts at every entry whose saturated sum differs from its left
  // neighbour's and ends at the next such entry.  A lane closes the runs
  // that start at its entries (the last one ends at the next lane's first
  // start), the lane with the chunk's first start also closes the run left
  // open by earlier chunks, and the chunk's spans are written after one
  // prefix sum.  Every entry read is reset to zero.
  SKC_HD bool acc_row(const Lanes& L, int y, int32_t* diff, int left, int lo, int hi) {
    if (y < row0 || y >= row1) return false;
    row_begin(L, y);
    constexpr int V = Lanes::n == 32 ? 4 : 1;
    constexpr int kNone = 0x7fffffff;
    int open_start = -1;   // warp-uniform: the run still open after a chunk
    int32_t open_v = 0;
    int32_t carry = 0;     // prefix sum before this chunk
    int32_t prev_sat = 0;  // saturated value of the entry before this chunk
    // Entries outside [lo, hi] are zero, so the chunks can start at a
    // multiple of V (16-byte loads); a chunk of zeros changes no sum and
    // starts no run, and is skipped after one load.
    const bool vec = V == 4 && ((uintptr_t)diff & 15) == 0;
    for (int base = vec ? (lo & ~(V - 1)) : lo; base < hi; base += Lanes::n * V) {
      const int i0 = base + L.lane * V;
      int32_t sat[V];
      if (vec && i0 + V <= hi) {
        const int4 q = *(const int4*)(diff + i0);
        sat[0] = q.x;
        sat[1 % V] = q.y;
        sat[2 % V] = q.z;
        sat[3 % V] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) sat[j] = i0 + j < hi ? diff[i0 + j] : 0;
      }
      bool nz = false;
#pragma unroll
      for (int j = 0; j < V; ++j) nz |= sat[j] != 0;
      if (!L.ballot(nz)) continue;
      if (nz) {
#pragma unroll
        for (int j = 0; j < V; ++j)
          if (i0 + j < hi) diff[i0 + j] = 0;
      }
      int32_t run = 0;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        run += sat[j];
        sat[j] = run;
      }
      const int32_t incl = LaneScanIncl(L, run);
      const int32_t pre = incl - run + carry;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int32_t v = sat[j] + pre;
        sat[j] = v > 255 ? 255 : v;
      }
      int32_t before = LaneBcast(L, sat[V - 1], L.lane > 0 ? L.lane - 1 : 0);
      if (L.lane == 0) before = prev_sat;
      unsigned bits = 0;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int32_t b = j == 0 ? before : sat[j - 1];
        if (i0 + j < hi && sat[j] != b) bits |= 1u << j;
      }
      const unsigned has = L.ballot(bits != 0);
      const int first_pos = bits ? i0 + Lanes::ffs(bits) - 1 : kNone;
      const unsigned later = has & ~((2u << L.lane) - 1u);
      int next_first = (int)L.shfl((uint32_t)first_pos, later ? Lanes::ffs(later) - 1 : L.lane);
      if (!later) next_first = kNone;
      // this lane's spans, in x order
      uint2 out[V + 1];
      int cnt = 0;
      unsigned long long fr = 0;
      auto put = [&](int s0, int w, int32_t a) {
        int x = left + s0, len = w;
        if (keep(x, y, len, (uint8_t)a)) {
          out[cnt++] = pack(x, len, (uint32_t)a);
          fr += (unsigned)len;
        }
      };
      if (has && open_start >= 0 && L.lane == Lanes::ffs(has) - 1)
        put(open_start, first_pos - open_start, open_v);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        if (!(bits & (1u << j))) continue;
        const unsigned rest = bits & ~((2u << j) - 1u);
        const int end = rest ? i0 + Lanes::ffs(rest) - 1 : next_first;
        if (end != kNone && sat[j] != 0) put(i0 + j, end - (i0 + j), sat[j]);
      }
      // the run left open: the chunk's last start, if any
      if (has) {
        const int src = 31 - clz_(has);
        const int lb = 31 - clz_(bits ? bits : 1u);
        const int32_t lv = sat[lb];
        const int lpos = i0 + lb;
        const int32_t v = LaneBcast(L, lv, Lanes::n == 32 ? src : 0);
        const int pos = LaneBcast(L, lpos, Lanes::n == 32 ? src : 0);
        open_start = v != 0 ? pos : -1;
        open_v = v;
      }
      const int32_t ci = LaneScanIncl(L, cnt);
      const uint32_t total = (uint32_t)LaneBcast(L, ci, Lanes::n - 1);
      if (total) {
        const uint32_t at = reserve(L, 0, total);
        uint2* dst = span_ptr(at + (uint32_t)(ci - cnt));
        if (dst) {
          for (int i = 0; i < cnt; ++i) dst[i] = out[i];
        }
        commit(L, total, fr);
      }
      carry += LaneBcast(L, incl, Lanes::n - 1);
      prev_sat = LaneBcast(L, sat[V - 1], Lanes::n - 1);
    }
    if (open_start >= 0) {
      int x = left + open_start, len = hi - open_start;
      if (keep(x, y, len, (uint8_t)open_v)) {
        const uint32_t at = reserve(L, 0, 1);
        if (!dead && L.leader()) pool[at] = pack(x, len, (uint32_t)open_v);
        commit(L, 1, L.leader() ? (unsigned)len : 0u);
      }
    }
    return true;
  }
};

template <typename Sink>
SKC_HD void InitPoolSink(const DevBatch& b, uint32_t p, const PassGeom& g, Sink* s) {
  const PassDesc pd = b.passes[p];
  const PassSweep sw = b.sweep[p];
  const CanvasDesc cd = b.canvases[pd.canvas];
  s->row0 = g.row0;
  s->row1 = g.row1;
  s->W = (int)cd.w;
  s->H = (int)cd.h;
  s->ga = pd.ga;
  s->srcover = (pd.flags & kPassSrcOver) != 0;
  s->raw = (pd.flags & kPassRawSpans) != 0;
  s->pool = b.spans;
  s->cap = b.span_cap < 0xFFFFFFFFull ? b.span_cap : 0xFFFFFFFFull;
  s->next = b.span_next;
  s->chunk = sw.chunk;
  s->rows = b.rowspan + sw.rbase;
  s->err = b.err;
  s->cur_row = kNaN32;
  s->row_start = s->cur = s->chunk_end = 0;
  s->dead = false;
  s->kept = 0;
  s->frags = 0;
}

template <typename Sink>
SKC_HD void FinishPass(const DevBatch& b, uint32_t p, Sink* s, const Lanes& L) {
  s->finish_row(L);
  const unsigned long long frags = LaneSum64(L, s->frags);
  L.sync();
  if (L.leader()) {
    b.pass_spans[p] = s->kept;
    if (b.pass_frags) b.pass_frags[p] = frags;
  }
}

SKC_HD void EmptyPass(const DevBatch& b, uint32_t p, const Lanes& L) {
  if (L.leader()) {
    b.pass_spans[p] = 0;
    if (b.pass_frags) b.pass_frags[p] = 0;
  }
}

// The generic sweep of pass p (LaneSweep, state in the pass's sweep memory).
template <typename Sink>
SKC_HDN void RunSweep(const DevBatch& b, uint32_t p, const PassGeom& g, Sink* sink,
                      const Lanes& lanes) {
  const PassDesc pd = b.passes[p];
  const PassSweep sw = b.sweep[p];
  SliceLayout L;
  L.compute(pd.cap, sizeof(Edge));
  const Edge* S = (const Edge*)(b.scratch + pd.slice_off + L.off[13]);
  int n = g.n_edges;
  SweepMem M = SweepMemAt(b.sweepmem + sw.work_off, n, g.acc_width);
  for (int i = lanes.lane; i < n; i += Lanes::n) M.W[i] = S[i];
  for (int i = lanes.lane; i <= g.acc_width; i += Lanes::n) M.diff[i] = 0;
  lanes.sync();
  LaneSweep<Sink> s;
  s.L = lanes;
  s.M = M;
  s.n = n;
  s.err = b.err;
  s.sink = sink;
  s.acc_left = g.acc_left;
  s.acc_width = g.acc_width;
  s.acc_y = kNaN32;
  s.touch_lo = 0x7fffffff;
  s.touch_hi = -1;
  s.scan_top = g.scan_top;
  s.walk((pd.flags & kPassEvenOdd) != 0, g.start_y, g.stop_y, g.left_bound, g.right_bound);
  s.flush_acc();
}

// Sweep of pass p through the generic sweep.  Row entries a register attempt
// may have written are cleared first.  kRaw: the pass may be a path clip's
// (raw spans); batches without path clips take the form without that test.
template <bool kRaw = true>
SKC_HDN void SweepPass(const DevBatch& b, uint32_t p, const Lanes& lanes) {
  const PassGeom g = b.geom[p];
  const int nrows = g.row1 - g.row0;
  if (g.n_edges <= 0 || nrows <= 0) {
    EmptyPass(b, p, lanes);
    return;
  }
  uint2* rows = b.rowspan + b.sweep[p].rbase;
  for (int r = lanes.lane; r < nrows; r += Lanes::n) rows[r] = make_uint2(0, 0);
  lanes.sync();
  PoolSinkT<kRaw> sink;
  InitPoolSink(b, p, g, &sink);
  RunSweep(b, p, g, &sink, lanes);
  FinishPass(b, p, &sink, lanes);
}

template <int M>
SKC_HD uint64_t RegSmemBytes(int32_t diff_cap) {
  return sizeof(RegSharedT<M>) + 4ull * (uint64_t)diff_cap;
}
// Accumulator entries of a pair in shared memory; wider passes keep theirs in
// their sweep memory.  The 32-edge form has room for some 1,024-pixel passes:
// with 3,072 entries the pairs of a 4,096-pixel canvas fill the shared memory
// before the registers (110,000 glyphs: 6.7 ms instead of 6.2); with 640, 400
// draws on 1204 pixels take 2.75 ms instead of 2.14.
template <int M>
SKC_HD int32_t PairDiffCap(int32_t diff_cap) {
  return M == 32 ? min_(diff_cap, 1156) : diff_cap;
}
template <int M>
SKC_HD uint64_t PairSmemBytes(int32_t diff_cap) {
  return sizeof(RegPairT<M>) + 4ull * (uint64_t)diff_cap;
}

// The accumulator of a register sweep, zeroed; it sits in shared memory when
// it fits.
SKC_HD void InitAcc(const DevBatch& b, uint32_t p, const PassGeom& g, const Lanes& lanes,
                    int32_t* sdiff, int32_t sdiff_cap, AccState* as) {
  const PassSweep sw = b.sweep[p];
  as->diff = g.acc_width + 1 <= sdiff_cap
                 ? sdiff
                 : SweepMemAt(b.sweepmem + sw.work_off, g.n_edges, g.acc_width).diff;
#pragma unroll 1
  for (int i = lanes.lane; i <= g.acc_width; i += Lanes::n) as->diff[i] = 0;
  as->left = g.acc_left;
  as->width = g.acc_width;
  as->shift = Lanes::n == 1 ? 0 : 5;
  while ((g.acc_width >> as->shift) >= 32) ++as->shift;
  as->y = kNaN32;
  as->touched = 0;
  as->flushing = false;
  lanes.sync();
}

// The walk of pass p (RegWalk); returns 0 when its active list outgrows the
// registers.
template <typename Sh, typename Hand>
SKC_HD int WalkPass(const DevBatch& b, uint32_t p, const PassGeom& g, const Lanes& lanes, Sh* sh,
                    Hand&& hand) {
  const PassDesc pd = b.passes[p];
  SliceLayout L;
  L.compute(pd.cap, sizeof(Edge));
  const Edge* S = (const Edge*)(b.scratch + pd.slice_off + L.off[13]);
  // rows whose coverage is kept (scan_top is a whole number)
  return RegWalk(lanes, *sh, S, g.n_edges, (pd.flags & kPassEvenOdd) != 0,
                 max_((int)g.scan_top, g.row0), g.row1, g.start_y, g.stop_y, g.left_bound, hand);
}

// Sweep of pass p through the register form of size M (kRaw: the pass may be a
// path clip's; batches without path clips take the form without that test).
// Returns false when its active list outgrows M after all: the caller then
// sweeps the pass with the generic form (SweepPass, which clears the rows the
// attempt wrote).  Walk and emission take turns here: the form for a caller
// without a second warp (the CPU build of the tests).
template <int M, bool kRaw = true>
SKC_HD bool SweepPassReg(const DevBatch& b, uint32_t p, const Lanes& lanes, RegSharedT<M>* sh,
                         int32_t* sdiff, int32_t sdiff_cap) {
  const PassGeom g = b.geom[p];
  if (g.n_edges <= 0 || g.row1 <= g.row0) {
    EmptyPass(b, p, lanes);
    return true;
  }
  // rows the sweep leaves without spans read as empty
  uint2* rows = b.rowspan + b.sweep[p].rbase;
#pragma unroll 1
  for (int r = lanes.lane; r < g.row1 - g.row0; r += Lanes::n) rows[r] = make_uint2(0, 0);
  lanes.sync();
  PoolSinkT<kRaw> sink;
  InitPoolSink(b, p, g, &sink);
  AccState as;
  InitAcc(b, p, g, lanes, sdiff, sdiff_cap, &as);
  if (!WalkPass(b, p, g, lanes, sh, [&](int nrec, bool last) {
        lanes.sync();
        RegEmit(lanes, *sh, sh->log[0], &sink, as, nrec, g.left_bound, g.right_bound, last);
        return &sh->log[0];
      })) {
    lanes.sync();
    return false;
  }
  FinishPass(b, p, &sink, lanes);
  return true;
}

// The same by two warps (the device's form): one walks and logs, the other
// emits the log before.  They meet() once a log, when the walker has filled
// one and the emitter is done with the other.  The emitter returns the pass's
// result.
template <int M, bool kRaw, typename Meet>
SKC_HD bool SweepPassPair(const DevBatch& b, uint32_t p, const Lanes& lanes, bool walker,
                          RegPairT<M>* sh, int32_t* sdiff, int32_t sdiff_cap, Meet&& meet) {
  const PassGeom g = b.geom[p];
  if (g.n_edges <= 0 || g.row1 <= g.row0) {
    if (!walker) EmptyPass(b, p, lanes);
    return true;
  }
  int buf = 0;
  if (walker) {
    auto hand = [&](int nrec, bool last) {
      if (lanes.leader()) {
        sh->filled[buf] = nrec;
        sh->filled[2 + buf] = last;
      }
      meet();
      buf ^= 1;
      return &sh->log[buf];
    };
    if (!WalkPass(b, p, g, lanes, sh, hand)) hand(-1, true);
    return true;
  }
  uint2* rows = b.rowspan + b.sweep[p].rbase;
#pragma unroll 1
  for (int r = lanes.lane; r < g.row1 - g.row0; r += Lanes::n) rows[r] = make_uint2(0, 0);
  lanes.sync();
  PoolSinkT<kRaw> sink;
  InitPoolSink(b, p, g, &sink);
  AccState as;
  InitAcc(b, p, g, lanes, sdiff, sdiff_cap, &as);
#pragma unroll 1
  for (;; buf ^= 1) {
    meet();
    const int nrec = sh->filled[buf];
    const bool last = sh->filled[2 + buf] != 0;
    if (nrec < 0) return false;
    RegEmit(lanes, *sh, sh->log[buf], &sink, as, nrec, g.left_bound, g.right_bound, last);
    if (last) break;
  }
  FinishPass(b, p, &sink, lanes);
  return true;
}



// ---------------------------------------------------------------------------
// StackBlur lines
// ---------------------------------------------------------------------------
SKC_HD int32_t StackBlurShr(int32_t r) {
  uint32_t d = (uint32_t)(r + 1) * (uint32_t)(r + 1);
  return (31 - clz_(d)) + 9;
}
SKC_HD uint64_t StackBlurMul(int32_t r) {
  uint64_t d = (uint64_t)(r + 1) * (uint64_t)(r + 1);
  return ((1ull << StackBlurShr(r)) + d - 1) / d;
}

// Blur one channel of a line of n pixels (`step` bytes apart) from src into
// dst (`out_step` bytes apart), both at the channel's first byte.  out0: the pixel value that the
// out_sum starts from -- the channel's own first one, or, in the vertical
// pass, slot 1's for slots 0 and 3 (sw_stack_blur.cc:175-179).  Sums are
// modulo the reference's 64 bits; Sum = int32_t where they stay below 2^31.
template <typename Sum>
SKC_HD void BlurChannelSums(const uint8_t* __restrict__ src, size_t step,
                            uint8_t* __restrict__ dst, size_t out_step, int n, int r, int out0) {
  const int rp1 = r + 1;
  const int nm1 = n - 1;
  const int64_t mul = (int64_t)StackBlurMul(r);
  const int shr = StackBlurShr(r);
  auto px = [&](int i) -> Sum { return (Sum)src[(size_t)i * step]; };
  Sum sum = px(0) * (Sum)(rp1 * (rp1 + 1) / 2), in_sum = 0, out_sum = (Sum)out0 * (Sum)rp1;
#pragma unroll 4
  for (int i = 1; i <= r; ++i) {
    const Sum v = px(min_(i, nm1));
    sum += v * (Sum)(rp1 - i);
    in_sum += v;
  }
#pragma unroll 4
  for (int i = 0; i < n; ++i) {
    const Sum out = px(max_(i - r, 0)), in = px(min_(i + rp1, nm1)), mid = px(min_(i + 1, nm1));
    // the low bits of the 64-bit product, whichever sign the sum has
    dst[(size_t)i * out_step] = (uint8_t)(((int64_t)sum * mul) >> shr);
    in_sum += in;
    sum += in_sum - out_sum;
    out_sum += mid - out;
    in_sum -= mid;
  }
}
SKC_HD void BlurChannel(const uint8_t* src, size_t step, uint8_t* dst, size_t out_step, int n,
                        int r, int out0) {
  // a wrong start of out_sum is off by at most 255 (r + 1), on every pixel
  if ((int64_t)(n + r + 1) * 255 * (r + 1) < (1ll << 31))
    BlurChannelSums<int32_t>(src, step, dst, out_step, n, r, out0);
  else
    BlurChannelSums<int64_t>(src, step, dst, out_step, n, r, out0);
}

// Blur one line of n pixels (stride in pixels) from src into dst (v: the
// vertical pass).
SKC_HDN void BlurLine(const uint8_t* src, uint8_t* dst, int n, size_t stride, int r, bool v) {
  for (int c = 0; c < 4; ++c)
    BlurChannel(src + c, 4 * stride, dst + c, 4 * stride, n, r,
                src[v && (c == 0 || c == 3) ? 1 : c]);
}

// Scalar composite of one row task (CPU execution of the pipeline; the GPU
// runs the warp-parallel form in kernels.cu with identical per-pixel order).
SKC_HDN void CompositeRowScalar(const DevBatch& b, const RowTask& rt, uint32_t* row) {
  const CanvasDesc cd = b.canvases[rt.canvas];
  const int y = (int)rt.y, x0 = (int)rt.x0, x1 = (int)rt.x1;
  uint32_t* gpx = (uint32_t*)(b.pixels + cd.px_off) + (size_t)y * cd.w + x0;
  for (int i = 0; i < x1 - x0; ++i) row[i] = cd.has_clear ? cd.clear_pm : RGBAtoARGB(gpx[i]);
  const uint32_t band = cd.band0 + ((uint32_t)y >> b.band_shift);
  for (uint32_t e = b.band_off[band]; e < b.band_off[band + 1]; ++e) {
    const PassComp pc = b.comp[b.bins[e]];
    if (y < pc.row0 || y >= pc.row1) continue;
    const uint2 rs = b.rowspan[pc.rbase + (y - pc.row0)];
    const Brush br = b.brushes[pc.brush];
    for (uint32_t s = rs.x; s < rs.x + rs.y; ++s) {
      uint2 sp = b.spans[s];
      int sx = (int)(sp.x & 0xFFFF), slen = (int)(sp.x >> 16);
      int xs = max_(sx, x0), xe = min_(sx + slen, x1);
      uint32_t alpha = sp.y & br.global_alpha;
      for (int x = xs; x < xe; ++x) {
        uint32_t c = BrushColor(br, x, y, b.stop_colors, b.stop_offsets, b.pixels, b.roundtrip,
                                b.conicals);
        if (alpha != 255) c = AlphaMulQ(c, alpha);
        if (br.cf_type) c = FilterColor(br, c, b.srgb_tables, b.cf_matrices);
        row[x - x0] = BlendPixel(row[x - x0], c, br.blend);
      }
    }
  }
  for (int i = 0; i < x1 - x0; ++i) gpx[i] = ARGBtoRGBA(row[i]);
}

}  // namespace skc

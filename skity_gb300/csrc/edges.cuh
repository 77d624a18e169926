// The geometry of one pass on one warp: Path -> QuadPath (-> stroke ->
// QuadPath) -> bounds -> fixed-point edges -> sort, with the lanes on
// different verbs, runs of a contour's segments, edges and sort positions.
// Every stage gives what the one-thread functions of geom.cuh, stroke.cuh and
// raster.cuh give (on the CPU the lanes are one thread); paths that are not
// regular (RegularVerb) go through those on one lane.
#pragma once
#include "kernels.cuh"
#include "stroke.cuh"
#include "sweep.cuh"

namespace skc {

// ---------------------------------------------------------------------------
// sort
// ---------------------------------------------------------------------------
// Scratch of one warp.  kSortKeys edges are sorted on chip, more in their
// pass's scratch slice.
constexpr int kSortKeys = 384;
struct SortKey {
  int32_t y, x, dx, idx;  // Edge::upper_y, x, dx; the edge
};
struct alignas(16) SortShared {
  int32_t first[64], last[64], depth[64];  // ranges still to partition
  int32_t l[64], r[64];                    // a partition's swaps
  SortKey keys[kSortKeys];
};

// SortEdges' order (sw_raster.cc:679-704).
struct SortKeyLess {
  SKC_HD bool operator()(const SortKey& a, const SortKey& b) const {
    return a.y != b.y ? a.y < b.y : a.x != b.x ? a.x < b.x : a.dx < b.dx;
  }
};

// Hoare partition of a[first, last) as std::sort makes it (median of three
// moved to `first`, unguarded scans), returning the cut.  The scans stop at
// the elements not below the pivot, from the left, and not above it, from the
// right; the k-th of one is swapped with the k-th of the other while they have
// not met.  So blocks are read from both ends, a ballot finds their stops, and
// as many as both have pending are swapped at once; what is left in the
// middle (less than two elements a lane) is finished the same way.
template <typename T, typename Less>
SKC_HD int PartitionLanes(const Lanes& L, SortShared* sh, T* a, int first, int last, Less less) {
  constexpr int NL = Lanes::n;
  {
    const int mid = first + (last - first) / 2;
    const T f = a[first], x = a[first + 1], y = a[mid], z = a[last - 1];
    int m;  // the median of x, y, z (median_to_first)
    if (less(x, y))
      m = less(y, z) ? mid : less(x, z) ? last - 1 : first + 1;
    else
      m = less(x, z) ? first + 1 : less(y, z) ? last - 1 : mid;
    L.sync();
    if (L.leader()) {
      a[first] = a[m];
      a[m] = f;
    }
    L.sync();
  }
  const T pivot = a[first];
  const unsigned le = (2u << L.lane) - 1u;
  int ln = first + 1, rn = last;  // not read yet: [ln, rn)
  int lb = 0, rb = 0;             // the blocks with pending stops
  unsigned lm = 0, rm = 0;
#pragma unroll 1
  for (;;) {
    if (!lm) {
      if (rn - ln < NL) break;
      lb = ln;
      lm = L.ballot(!less(a[lb + L.lane], pivot));
      ln += NL;
      continue;
    }
    if (!rm) {
      if (rn - ln < NL) break;
      rn -= NL;
      rb = rn;
      rm = L.ballot(!less(pivot, a[rb + L.lane]));
      continue;
    }
    const int k = min_(Lanes::popc(lm), Lanes::popc(rm));
    const bool inl = (lm >> L.lane) & 1u, inr = (rm >> L.lane) & 1u;
    const int rl = Lanes::popc(lm & L.lt_mask()), rr = Lanes::popc(rm & ~le);
    if (inl && rl < k) sh->l[rl] = lb + L.lane;
    if (inr && rr < k) sh->r[rr] = rb + L.lane;
    L.sync();
    if (L.lane < k) {
      const int i = sh->l[L.lane], j = sh->r[L.lane];
      const T t = a[i];
      a[i] = a[j];
      a[j] = t;
    }
    lm = L.ballot(inl && rl >= k);
    rm = L.ballot(inr && rr >= k);
    L.sync();
  }
  const int a0 = lm ? lb + Lanes::ffs(lm) - 1 : ln;
  const int a1 = rm ? rb + 32 - clz_(rm) : rn;
  const int p0 = a0 + L.lane, p1 = p0 + NL;
  const bool l0 = p0 < a1 && !less(a[p0], pivot), l1 = p1 < a1 && !less(a[p1], pivot);
  const bool r0 = p0 < a1 && !less(pivot, a[p0]), r1 = p1 < a1 && !less(pivot, a[p1]);
  const unsigned ml0 = L.ballot(l0), ml1 = L.ballot(l1), mr0 = L.ballot(r0), mr1 = L.ballot(r1);
  const int cl = Lanes::popc(ml0) + Lanes::popc(ml1), cr = Lanes::popc(mr0) + Lanes::popc(mr1);
  if (l0) sh->l[Lanes::popc(ml0 & L.lt_mask())] = p0;
  if (l1) sh->l[Lanes::popc(ml0) + Lanes::popc(ml1 & L.lt_mask())] = p1;
  if (r1) sh->r[Lanes::popc(mr1 & ~le)] = p1;
  if (r0) sh->r[Lanes::popc(mr1) + Lanes::popc(mr0 & ~le)] = p0;
  L.sync();
  int m = 0;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const int r = k * NL + L.lane;
    const bool swap = r < min_(cl, cr) && sh->l[r] < sh->r[r];
    if (swap) {
      const int i = sh->l[r], j = sh->r[r];
      const T t = a[i];
      a[i] = a[j];
      a[j] = t;
    }
    m += Lanes::popc(L.ballot(swap));
  }
  // where the left scan stops next: its next stop, or what the last swap put
  // on the right, or the first element already read there
  const int cut = min_(m < cl ? sh->l[m] : a1, m > 0 ? sh->r[m - 1] : a1);
  L.sync();
  return cut;
}

// The partitioning loop of introsort: afterwards a[0, n) is in blocks of at
// most 16 elements (or heap-sorted ones), none below an earlier block's, and a
// stable sort of it (the final insertion sort) finishes.
template <typename T, typename Less>
SKC_HD void IntrosortPartitions(const Lanes& L, SortShared* sh, T* a, int n, Less less) {
  if (n <= 16) return;
  int sp = 0;
  int first = 0, last = n, depth = 2 * (31 - clz_((uint32_t)n));
#pragma unroll 1
  for (;;) {
    if (last - first > 16 && depth > 0 && sp < 64) {
      const int cut = PartitionLanes(L, sh, a, first, last, less);
      --depth;
      if (L.leader()) {
        sh->first[sp] = first;
        sh->last[sp] = cut;
        sh->depth[sp] = depth;
      }
      ++sp;
      first = cut;
      continue;
    }
    if (last - first > 16) {
      if (L.leader()) heap_sort_range(a + first, last - first, less);
      L.sync();
    }
    if (sp == 0) break;
    --sp;
    L.sync();
    first = sh->first[sp];
    last = sh->last[sp];
    depth = sh->depth[sp];
    L.sync();
  }
}

// The place of a[i] in the stable sort that finishes (at most 15 away).
template <typename T, typename Less>
SKC_HD int StableRank(const T* a, int n, int i, Less less) {
  const T v = a[i];
  int r = i;
#pragma unroll 1
  for (int d = 1; d < 16; ++d) {
    if (i - d >= 0 && less(v, a[i - d])) --r;
    if (i + d < n && less(a[i + d], v)) ++r;
  }
  return r;
}

// ---------------------------------------------------------------------------
// QuadPath
// ---------------------------------------------------------------------------
SKC_HD int VerbPoints(uint8_t v) { return v == kClose ? 0 : v >= kCubic ? 3 : (v + 2) / 2; }
SKC_HD bool IsSegment(uint8_t v) { return v != kMove && v != kClose; }

// Where a warp's verbs stand in their path: points before each, the last
// MoveTo's point, the verb before; carried from 32 verbs to the next.
struct VerbWalk {
  int np = 0;        // points before the chunk
  int move = 0;      // the last MoveTo's point
  uint8_t last = kDone;
  // this lane's verb
  uint8_t verb, prev;
  int p;             // its first point
  int contour;       // its contour's MoveTo point (a MoveTo's: the one before)
  SKC_HD void load(const Lanes& L, const PathView& q, int base) {
    constexpr int NL = Lanes::n;
    const int i = base + L.lane;
    verb = i < q.nv ? q.verbs[i] : (uint8_t)kClose;
    const int pc = i < q.nv ? VerbPoints(verb) : 0;
    const int incl = LaneScanIncl(L, pc);
    p = np + incl - pc;
    int mv = i < q.nv && verb == kMove ? p : -1;
#ifdef SKC_WARP_LANES
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, mv, o);
      if (L.lane >= o) mv = max_(mv, t);
    }
    const int before = __shfl_up_sync(0xffffffffu, mv, 1);
    contour = L.lane == 0 || before < 0 ? move : before;
    const int pv = __shfl_up_sync(0xffffffffu, (int)verb, 1);
    prev = L.lane == 0 ? last : (uint8_t)pv;
#else
    contour = move;
    prev = last;
#endif
    np += LaneBcast(L, incl, NL - 1);
    move = max_(move, LaneBcast(L, mv, NL - 1));
    last = (uint8_t)LaneBcast(L, (int)verb, NL - 1);
  }
};

// Whether verb i stands where a regular path has it: contours are a MoveTo,
// segments and at most one Close -- what Path's own calls build, but for empty
// contours.
SKC_HD bool RegularVerb(const VerbWalk& w, int i, int nv) {
  if (w.verb == kMove) return !(i > 0 && w.prev == kMove) && i != nv - 1;
  const bool after_seg = i > 0 && IsSegment(w.prev);
  if (w.verb == kClose) return after_seg;
  return after_seg || (i > 0 && w.prev == kMove);
}

// Stroke::QuadPath (QuadPath, geom.cuh) on a warp.  A regular path's verbs
// have their output known from the verb itself: lines and quads as they are, a
// conic's two quads, a cubic's n, and a Close after the line back to the
// contour's start (PathIter::AutoClose).  Other paths go through the
// one-thread form.
SKC_HDN void QuadPathSolo(const Lanes& L, const PathView& src, DPath* dst) {
  if (L.leader()) QuadPath(src, dst);
  L.sync();
  dst->nv = LaneBcast(L, dst->nv, 0);
  dst->np = LaneBcast(L, dst->np, 0);
  dst->nw = LaneBcast(L, dst->nw, 0);
}
SKC_HDN void QuadPathLanes(const Lanes& L, const PathView& src, DPath* dst) {
  constexpr int NL = Lanes::n;
  bool odd = false;
  {
    VerbWalk w;
#pragma unroll 1
    for (int base = 0; base < src.nv; base += NL) {
      w.load(L, src, base);
      const int i = base + L.lane;
      if (i < src.nv) odd = odd || !RegularVerb(w, i, src.nv);
    }
  }
  if (L.ballot(odd)) {
    QuadPathSolo(L, src, dst);
    return;
  }
  int nv = 0, np = 0, wi = 0;
  VerbWalk w;
#pragma unroll 1
  for (int base = 0; base < src.nv; base += NL) {
    w.load(L, src, base);
    const bool valid = base + L.lane < src.nv;
    const int conic = valid && w.verb == kConic ? 1 : 0;
    const int winc = LaneScanIncl(L, conic);
    P pts[4];
    int ov = 0, op = 0;
    double n = 0;
    if (valid) {
      if (w.verb == kClose) {
        // back to the contour's start: a line unless there (or not a number)
        pts[0] = src.pts[w.p - 1];
        pts[1] = src.pts[w.contour];
        const bool line = !PEq(pts[0], pts[1]) && !(isnan_(pts[0].x) || isnan_(pts[0].y) ||
                                                   isnan_(pts[1].x) || isnan_(pts[1].y));
        ov = line ? 2 : 1;
        op = line ? 1 : 0;
      } else {
        const int k = VerbPoints(w.verb);
        pts[0] = w.verb == kMove ? src.pts[w.p] : src.pts[w.p - 1];
        if (w.verb != kMove)
          for (int j = 0; j < k; ++j) pts[1 + j] = src.pts[w.p + j];
        ov = 1;
        op = k;
        if (w.verb == kConic) {
          ov = 2;
          op = 4;
        } else if (w.verb == kCubic) {
          n = CubicQuadCountD(pts);
          int c = 0;
          while (c < n) ++c;  // quads of `for (i = 0; i < n; ++i)`
          ov = c;
          op = 2 * c;
        }
      }
    }
    const int iv = LaneScanIncl(L, ov), ip = LaneScanIncl(L, op);
    int vo = nv + iv - ov, po = np + ip - op;
    auto put_v = [&](uint8_t v) {
      if (vo < dst->cap_v) dst->verbs[vo] = v;
      ++vo;
    };
    auto put_p = [&](P q) {
      if (po < dst->cap_p) dst->pts[po] = q;
      ++po;
    };
    if (valid) {
      if (w.verb == kClose) {
        if (ov == 2) {
          put_v(kLine);
          put_p(pts[1]);
        }
        put_v(kClose);
      } else if (w.verb == kConic) {
        P q[5];
        ConicTo2Quads(pts[0], pts[1], pts[2], src.w[wi + winc - 1], q);
        for (int j = 1; j < 5; ++j) {
          if (j & 1) put_v(kQuad);
          put_p(q[j]);
        }
      } else if (w.verb == kCubic) {
        CubicCoeff cc;
        cc.set(pts[0], pts[1], pts[2], pts[3]);
        QuadCoeff qc;
        qc.set(mkP(3.f * (pts[1].x - pts[0].x), 3.f * (pts[1].y - pts[0].y)),
               mkP(3.f * (pts[2].x - pts[1].x), 3.f * (pts[2].y - pts[1].y)),
               mkP(3.f * (pts[3].x - pts[2].x), 3.f * (pts[3].y - pts[2].y)));
#pragma unroll 1
        for (int i = 0; i < ov; ++i) {
          P q[3];
          CubicQuadAt(pts, cc, qc, n, i, q);
          put_v(kQuad);
          put_p(q[1]);
          put_p(q[2]);
        }
      } else {
        put_v(w.verb);
        if (w.verb == kMove) put_p(pts[0]);
        if (w.verb != kMove)
          for (int j = 0; j < op; ++j) put_p(pts[1 + j]);
      }
    }
    nv += LaneBcast(L, iv, NL - 1);
    np += LaneBcast(L, ip, NL - 1);
    wi += LaneBcast(L, winc, NL - 1);
  }
  dst->nv = nv;
  dst->np = np;
  dst->nw = 0;
  L.sync();
}

// ---------------------------------------------------------------------------
// stroker
// ---------------------------------------------------------------------------
SKC_HD float LaneBcastF(const Lanes& L, float v, int src) {
#ifdef SKC_WARP_LANES
  return __shfl_sync(0xffffffffu, v, src);
#else
  return v;
#endif
}
SKC_HD P LaneBcastP(const Lanes& L, P p, int src) {
  return mkP(LaneBcastF(L, p.x, src), LaneBcastF(L, p.y, src));
}

// A builder that goes on behind (v, p, w) elements of `base`, inside a contour.
SKC_HD DPath PathTail(const DPath& base, int v, int p, int w) {
  DPath d;
  d.init(base.verbs + v, max_(base.cap_v - v, 0), base.pts + p, max_(base.cap_p - p, 0), base.w + w,
         max_(base.cap_w - w, 0));
  d.last_move = 0;
  d.last_verb = kLine;
  return d;
}

// Stroke::StrokePath (StrokePath, stroke.cuh) on a warp, for the paths
// QuadPathLanes calls regular.  Each contour's segments are dealt to the lanes
// in runs; a lane's stroker starts behind a segment whose end normals are its
// own (EndNormals, twice in a row: the second's start is then the path's
// point), so it joins and offsets its run as the one stroker would.  A walk
// drafts each run's outline in the lane's share of `draft` and counts it, and
// the lanes copy their drafts to where the runs before them end (a draft that
// does not fit: a second walk writes there); the contour's end -- join or
// caps, the inner side reversed -- follows.
// A quad that is not resolved within the depth limit leaves its depth to the
// quads after it: runs behind one are counted again from that depth.
// `pidx`: room for an int per verb; `draft`: room for the runs' outlines, 16
// bytes aligned.  False: not that kind of path, or depths that have not
// settled; the caller strokes it on one lane.  The stroker's chain of
// arithmetic is what bounds it, and a counting walk before the writing one was
// as long: geometry of 305 long strokes and fills 5.6 -> 4.6 ms, of 400 effects
// draws 0.41 -> 0.28, of an 8-pass icon 0.108 -> 0.082.
SKC_HDN bool StrokePathLanes(const Lanes& L, const PathView& src, float width, float miter,
                             int cap, int join, DPath* outer, DPath* inner, int inner_max[3],
                             int32_t* pidx, uint8_t* draft, uint64_t draft_bytes) {
  constexpr int NL = Lanes::n;
  // a lane's draft: two sides of `room` points, weights and verbs each
  const uint64_t share = draft_bytes / (2 * NL) & ~(uint64_t)15;
  const int room = (int)(share / 13 < (1u << 28) ? share / 13 : 1u << 28);
  DPath drafts[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint8_t* at = draft + (2 * L.lane + k) * share;
    drafts[k].init(at + 12ull * room, room, (P*)at, room, (float*)(at + 8ull * room), room);
  }
  {
    bool odd = false;
    VerbWalk w;
#pragma unroll 1
    for (int base = 0; base < src.nv; base += NL) {
      w.load(L, src, base);
      const int i = base + L.lane;
      if (i < src.nv) {
        pidx[i] = w.p;
        odd = odd || !RegularVerb(w, i, src.nv) ||
              (w.verb != kMove && w.verb != kClose && w.verb != kLine && w.verb != kQuad);
      }
    }
    if (L.ballot(odd)) return false;
  }
  L.sync();
  int ov = 0, op = 0, ow = 0;  // the outline so far
  inner_max[0] = inner_max[1] = inner_max[2] = 0;
  int depth = 0;         // Stroker::recursion_depth between contours
  bool settled = false;
#pragma unroll 1
  for (int v0 = 0; v0 < src.nv;) {
    // the contour: a MoveTo, the segments [s0, s1), a Close or not
    const int s0 = v0 + 1;
    int s1 = src.nv;
#pragma unroll 1
    for (int base = s0; base < src.nv; base += NL) {
      const int i = base + L.lane;
      const unsigned end = L.ballot(i < src.nv && !IsSegment(src.verbs[i]));
      if (end) {
        s1 = base + Lanes::ffs(end) - 1;
        break;
      }
    }
    const bool close = s1 < src.nv && src.verbs[s1] == kClose;
    v0 = close ? s1 + 1 : s1;
    const P start = src.pts[pidx[s0 - 1]];
    if (close) {  // behind the line back to the start (PathIter::AutoClose)
      const P end = src.pts[pidx[s1] - 1];
      if (!PEq(end, start) &&
          !(isnan_(end.x) || isnan_(end.y) || isnan_(start.x) || isnan_(start.y)))
        ++s1;
    }
    auto is_quad = [&](int i) { return src.verbs[i] == kQuad; };  // (a Close is a line)
    auto points = [&](int i) { return src.verbs[i] == kClose ? &start : src.pts + pidx[i]; };

    // this lane's run [a, e)
    Stroker st;
    st.init(width * 0.5f, miter, cap, join, nullptr, nullptr);
    const int per = (s1 - s0 + NL - 1) / NL;
    int a = min_(s0 + L.lane * per, s1);
    st.segment_count = 0;
    st.first_pt = st.prev_pt = start;
    auto ends = [&](int i, P* n, P* u) {
      return st.EndNormals(src.pts[pidx[i] - 1], is_quad(i), points(i), n, u);
    };
    if (a > s0) {
#pragma unroll 1
      for (; a < s1; ++a) {
        P n, u;
        if (a - 2 >= s0 && !ends(a - 2, &n, &u)) continue;
        if (!ends(a - 1, &n, &u)) continue;
        st.segment_count = 1;
        st.join_completed = true;
        st.prev_pt = src.pts[pidx[a] - 1];
        st.prev_normal = n;
        st.prev_unit_normal = u;
        break;
      }
    }
    int e = s1;
#ifdef SKC_WARP_LANES
    {  // runs end where the next one starts
      const int t = __shfl_down_sync(0xffffffffu, a, 1);
      if (L.lane < 31) e = t;
    }
#endif
    Stroker from = st;
    DPath o, in;
    int n[6], at[6];  // the run's elements and its place: verbs, points, weights of both sides
    from.recursion_depth = depth;
#pragma unroll 1
    for (int walk = 0;; ++walk) {
      // drafting walks, until the depths agree; then, if need be, one that
      // writes
      const bool write = walk > 0 && settled;
      if (write) {
        o = PathTail(*outer, ov + at[0], op + at[1], ow + at[2]);
        in = PathTail(*inner, at[3], at[4], at[5]);
      } else {
        o = PathTail(drafts[0], 0, 0, 0);
        in = PathTail(drafts[1], 0, 0, 0);
      }
      st = from;
      st.outer = &o;
      st.inner = &in;
#pragma unroll 1
      for (int i = a; i < e; ++i) {
        const P* q = points(i);
        if (is_quad(i))
          st.QuadTo(q[0], q[1]);
        else
          st.LineTo(q[0]);
      }
      if (write) break;
      const int before = LanePrev(L, st.recursion_depth, depth);
      settled = L.ballot(before != from.recursion_depth) == 0;
      from.recursion_depth = before;
      if (!settled) {
        if (walk == 3) return false;
        continue;
      }
      n[0] = o.nv, n[1] = o.np, n[2] = o.nw, n[3] = in.nv, n[4] = in.np, n[5] = in.nw;
#pragma unroll
      for (int k = 0; k < 6; ++k) at[k] = LaneScanIncl(L, n[k]) - n[k];
      if (!L.ballot(o.overflow() || in.overflow())) {
        auto copy = [](auto* to, int first, int cap_, const auto* from_, int count) {
          const int fit = min_(count, cap_ - first);
#pragma unroll 4
          for (int k = 0; k < fit; ++k) to[first + k] = from_[k];
        };
        copy(outer->pts, op + at[1], outer->cap_p, o.pts, n[1]);
        copy(inner->pts, at[4], inner->cap_p, in.pts, n[4]);
        copy(outer->verbs, ov + at[0], outer->cap_v, o.verbs, n[0]);
        copy(inner->verbs, at[3], inner->cap_v, in.verbs, n[3]);
        copy(outer->w, ow + at[2], outer->cap_w, o.w, n[2]);
        copy(inner->w, at[5], inner->cap_w, in.w, n[5]);
        break;
      }
    }
    settled = false;
    depth = LaneBcast(L, st.recursion_depth, NL - 1);
    L.sync();
    // the contour's end, by the last lane that has a run (its state is the
    // stroker's) with the first lane's first segment
    const int last = Lanes::n == 32 ? 31 - clz_(L.ballot(a < e) | 1u) : 0;
    st.segment_count = LaneBcast(L, st.segment_count, last);
    st.prev_pt = LaneBcastP(L, st.prev_pt, last);
    st.prev_normal = LaneBcastP(L, st.prev_normal, last);
    st.prev_unit_normal = LaneBcastP(L, st.prev_unit_normal, last);
    st.first_normal = LaneBcastP(L, st.first_normal, 0);
    st.first_unit_normal = LaneBcastP(L, st.first_unit_normal, 0);
    st.first_outer_pt = LaneBcastP(L, st.first_outer_pt, 0);
    const int in_lane = Lanes::n == 32 ? 31 - clz_(L.ballot(n[4] > 0) | 1u) : 0;
    const P in_last = LaneBcastP(L, in.last_pt, in_lane);
    int tot[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) tot[k] = LaneBcast(L, at[k] + n[k], NL - 1);
    int iv = tot[3], ip = tot[4], iw = tot[5];
    ov += tot[0];
    op += tot[1];
    ow += tot[2];
    if (st.segment_count > 0) {
      // every lane makes the same few elements (the same values are stored)
      o = PathTail(*outer, ov, op, ow);
      in = PathTail(*inner, iv, ip, iw);
      in.last_pt = in_last;
      st.outer = &o;
      st.inner = &in;
      if (close) {
        st.Join(join == kMiterJoin && miter <= 1.f ? (int)kBevelJoin : join, &o, &in,
                st.prev_unit_normal, st.prev_pt, st.first_unit_normal);
        o.pushv(kClose);
        o.MoveTo(in.last_pt);
      } else {
        st.Cap(&o, st.prev_pt, st.prev_normal, in.last_pt);
      }
      iv += in.nv;
      ip += in.np;
      iw += in.nw;
      ov += o.nv;
      op += o.np;
      ow += o.nw;
      L.sync();
      // Path::ReversePathTo(inner): its segments last to first, its points
      // from the one before the last
      if (inner->cap_v >= iv && inner->cap_p >= ip && inner->cap_w >= iw) {
#pragma unroll 1
        for (int k = L.lane; k < iv - 1; k += NL)
          if (ov + k < outer->cap_v) outer->verbs[ov + k] = inner->verbs[iv - 1 - k];
#pragma unroll 1
        for (int k = L.lane; k < ip - 1; k += NL)
          if (op + k < outer->cap_p) outer->pts[op + k] = inner->pts[ip - 2 - k];
#pragma unroll 1
        for (int k = L.lane; k < iw; k += NL)
          if (ow + k < outer->cap_w) outer->w[ow + k] = inner->w[iw - 1 - k];
      }
      ov += iv - 1;
      op += ip - 1;
      ow += iw;
      o = PathTail(*outer, ov, op, ow);
      if (!close)
        st.Cap(&o, st.first_pt, mkP(-st.first_normal.x, -st.first_normal.y), st.first_outer_pt);
      o.pushv(kClose);
      ov += o.nv;
      op += o.np;
      ow += o.nw;
      L.sync();
    }
    inner_max[0] = max_(inner_max[0], iv);
    inner_max[1] = max_(inner_max[1], ip);
    inner_max[2] = max_(inner_max[2], iw);
  }
  outer->nv = ov;
  outer->np = op;
  outer->nw = ow;
  return true;
}

// ---------------------------------------------------------------------------
// bounds and edges
// ---------------------------------------------------------------------------
SKC_HD float LaneMinF(const Lanes& L, float v) {
#ifdef SKC_WARP_LANES
  for (int o = 16; o > 0; o >>= 1) v = min_(v, __shfl_xor_sync(0xffffffffu, v, o));
#endif
  return v;
}
SKC_HD float LaneMaxF(const Lanes& L, float v) {
#ifdef SKC_WARP_LANES
  for (int o = 16; o > 0; o >>= 1) v = max_(v, __shfl_xor_sync(0xffffffffu, v, o));
#endif
  return v;
}

// Pixel-space bounds of a mapped quad path and the scan bounds derived from
// them (sw_raster.cc:731-754, path.cc:1341-1360).  Every lane starts from the
// first point, so a point that is not a number is passed by, as in one
// thread's walk, and kept if it is the first.
SKC_HD RasterBounds BoundsLanes(const Lanes& L, const PathView& q, const Xform& xf, float cl,
                                float ct, float cr, float cb) {
  int n = q.np;
  if (q.nv > 1 && q.verbs[q.nv - 1] == kMove) n--;
  float l = 0, t = 0, r = 0, b = 0;
  if (n > 0) {
    const P p0 = xf.map(q.pts[0]);
    l = r = p0.x;
    t = b = p0.y;
#pragma unroll 1
    for (int i = 1 + L.lane; i < n; i += Lanes::n) {
      const P pi = xf.map(q.pts[i]);
      l = min_(l, pi.x);
      r = max_(r, pi.x);
      t = min_(t, pi.y);
      b = max_(b, pi.y);
    }
    l = LaneMinF(L, l);
    r = LaneMaxF(L, r);
    t = LaneMinF(L, t);
    b = LaneMaxF(L, b);
  }
  return ScanBounds(n > 0, l, t, r, b, cl, ct, cr, cb);
}

// SWEdgeBuilder::BuildEdges over PathEdgeIter (sw_edge.cc:299-336,
// src/graphic/path_priv.hpp:75-170): every segment of the quad path, and the
// line that closes each contour at its Close, at the next MoveTo or at the
// path's end.  Points are mapped by the canvas matrix first (Xform).  A lane
// takes a verb and its at most two edges; they keep the path's order.  Returns
// the number of edges (may exceed cap: only cap are stored).
SKC_HDN int BuildEdgesLanes(const Lanes& L, const PathView& q, const Xform& xf, float top,
                            float bottom, Edge* out, int cap) {
  constexpr int NL = Lanes::n;
  const Fixed y_top = ScanFixed(top), y_bottom = ScanFixed(bottom);
  int total = 0;
  VerbWalk w;
#pragma unroll 1
  for (int base = 0; base <= q.nv; base += NL) {  // one past the end: the last contour's close
    w.load(L, q, base);
    const int i = base + L.lane;
    P seg[5];
    int count = 0;     // edges before those outside the scan are dropped
    bool quad = false;
    if (i <= q.nv) {
      if (i == q.nv || !IsSegment(w.verb)) {
        if (i > 0 && IsSegment(w.prev)) {
          seg[0] = xf.map(q.pts[w.p - 1]);
          seg[1] = xf.map(q.pts[w.contour]);
          count = 1;
        }
      } else if (w.verb == kLine) {
        seg[0] = xf.map(q.pts[w.p - 1]);
        seg[1] = xf.map(q.pts[w.p]);
        count = 1;
      } else if (w.verb == kQuad) {
        const P s[3] = {xf.map(q.pts[w.p - 1]), xf.map(q.pts[w.p]), xf.map(q.pts[w.p + 1])};
        count = 1 + ChopQuadAtYExtrema(s, seg);
        quad = true;
      }
    }
    bool keep0 = false, keep1 = false;
    if (count > 0) keep0 = quad ? QuadKept(seg, y_top, y_bottom) : LineKept(seg[0], seg[1], y_top, y_bottom);
    if (count > 1) keep1 = QuadKept(seg + 2, y_top, y_bottom);
    const int mine = (keep0 ? 1 : 0) + (keep1 ? 1 : 0);
    const int incl = LaneScanIncl(L, mine);
    int at = total + incl - mine;
#pragma unroll 1
    for (int j = 0; j < mine; ++j) {
      const bool second = j == 1 || !keep0;
      Edge e;
      if (quad) {
        const P s[3] = {second ? seg[2] : seg[0], second ? seg[3] : seg[1], second ? seg[4] : seg[2]};
        SetQuad(&e, s);
      } else {
        SetLine(&e, seg[0], seg[1]);
      }
      if (at < cap) out[at] = e;
      ++at;
    }
    total += LaneBcast(L, incl, NL - 1);
  }
  L.sync();
  return total;
}

// ---------------------------------------------------------------------------
// the passes
// ---------------------------------------------------------------------------
SKC_HD PathView PassPath(const DevBatch& b, const PassDesc& pd) {
  const DrawDesc dd = b.draws[pd.draw];
  PathView src;
  src.verbs = b.verbs + dd.v0;
  src.pts = b.pts + dd.p0;
  src.w = b.weights + dd.w0;
  src.nv = (int)dd.nv;
  src.np = (int)dd.np;
  src.nw = (int)dd.nw;
  return src;
}

// The outline of a stroked pass into its scratch slice: QuadPath of the path,
// then the stroker.  PassGeom gets the sizes (status 1: one did not fit).
SKC_HDN void StrokePass(const DevBatch& b, uint32_t p, const Lanes& L) {
  const PassDesc pd = b.passes[p];
  if (!(pd.flags & kPassStroke)) return;
  SliceLayout S;
  S.compute(pd.cap, sizeof(Edge));
  uint8_t* base = b.scratch + pd.slice_off;
  DPath q1;
  q1.init(base + S.off[0], pd.cap[0], (P*)(base + S.off[1]), pd.cap[1], (float*)(base + S.off[2]),
          pd.cap[2]);
  QuadPathLanes(L, PassPath(b, pd), &q1);
  DPath outer, inner;
  outer.init(base + S.off[3], pd.cap[3], (P*)(base + S.off[4]), pd.cap[4],
             (float*)(base + S.off[5]), pd.cap[5]);
  inner.init(base + S.off[6], pd.cap[6], (P*)(base + S.off[7]), pd.cap[7],
             (float*)(base + S.off[8]), pd.cap[8]);
  int imax[3] = {0, 0, 0};
  const bool fits = !q1.overflow();
  const int cap = (int)(pd.cap_join & 0xFF), join = (int)(pd.cap_join >> 8);
  if (fits && !StrokePathLanes(L, q1.view(), pd.stroke_width, pd.miter, cap, join, &outer, &inner,
                               imax, (int32_t*)(base + S.off[14]), base + S.off[12],
                               S.off[14] - S.off[12])) {
    outer.reset();
    inner.reset();
    if (L.leader())
      StrokePath(q1.view(), pd.stroke_width, pd.miter, cap, join, &outer, &inner, imax);
  }
  if (!L.leader()) return;
  PassGeom& g = b.geom[p];
  g.n_edges = g.row0 = g.row1 = 0;
  g.need[0] = q1.nv;
  g.need[1] = q1.np;
  g.need[2] = q1.nw;
  g.need[3] = outer.nv;
  g.need[4] = outer.np;
  g.need[5] = outer.nw;
  g.need[6] = imax[0];
  g.need[7] = imax[1];
  g.need[8] = imax[2];
  for (int k = 9; k < 13; ++k) g.need[k] = 0;
  g.status = !fits || outer.overflow() || imax[0] > pd.cap[6] || imax[1] > pd.cap[7] ||
                     imax[2] > pd.cap[8]
                 ? 1
                 : 0;
}

// A bound of the sweep's active list: an edge joins it at upper_y and leaves
// after its last piece, so the list never holds more edges than the largest
// overlap of the [upper_y, last y) ranges -- at some edge's start, the edges
// up to it that end later.  S[0, n) sorted; tmp: room for 2 n words.
SKC_HD int MaxActive(const Lanes& L, SortShared* sh, const Edge* S, int n, int32_t* tmp) {
  constexpr int NL = Lanes::n;
  const bool few = n <= 256;
  int32_t* low = few ? (int32_t*)sh->keys : tmp;
#pragma unroll 1
  for (int i = L.lane; i < n; i += NL)
    low[i] = S[i].curve_count != 0 ? max_(S[i].lower_y, S[i].q_last_y) : S[i].lower_y;
  L.sync();
  int best = 0;
  if (few) {  // count the ends past each start
#pragma unroll 1
    for (int base = 0; base < n; base += NL) {
      const int i = base + L.lane;
      const int32_t u = i < n ? S[i].upper_y : 0;
      int c = 0;
      const int end = min_(base + NL, n);
#pragma unroll 4
      for (int j = 0; j < end; ++j) c += (j <= i && low[j] > u) ? 1 : 0;
      if (i < n) best = max_(best, c);
    }
  } else {    // sort the ends and search them
    IntLess less;
    IntrosortPartitions(L, sh, low, n, less);
    int32_t* sorted = tmp + n;
#pragma unroll 1
    for (int i = L.lane; i < n; i += NL) sorted[StableRank(low, n, i, less)] = low[i];
    L.sync();
#pragma unroll 1
    for (int i = L.lane; i < n; i += NL) {
      const int32_t u = S[i].upper_y;
      int lo = 0, hi = n;  // ends at or before u
#pragma unroll 1
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sorted[mid] <= u) lo = mid + 1;
        else hi = mid;
      }
      best = max_(best, i + 1 - lo);
    }
  }
  return LaneMax(L, best);
}

// The rest of a pass's geometry: QuadPath of its path (of its outline, when
// stroked), bounds, edges, sort; writes PassGeom.
SKC_HDN void EdgesPass(const DevBatch& b, uint32_t p, const Lanes& L, SortShared* sh) {
  constexpr int NL = Lanes::n;
  const PassDesc pd = b.passes[p];
  const bool stroke = (pd.flags & kPassStroke) != 0;
  PassGeom g;
  g.status = 0;
  g.n_edges = 0;
  g.start_y = g.stop_y = 0;
  g.left_bound = g.right_bound = 0;
  g.acc_left = g.acc_width = 0;
  g.scan_top = 0;
  g.row0 = g.row1 = 0;
  g.raw_spans = (pd.flags & kPassRawSpans) != 0 ? 1 : 0;
  g.max_active = 0;
  for (int k = 0; k < 13; ++k) g.need[k] = 0;
  auto done = [&]() {
    if (L.leader()) b.geom[p] = g;
  };
  SliceLayout S;
  S.compute(pd.cap, sizeof(Edge));
  uint8_t* base = b.scratch + pd.slice_off;
  PathView src;
  if (stroke) {
    g.status = b.geom[p].status;
    for (int k = 0; k < 9; ++k) g.need[k] = b.geom[p].need[k];
    L.sync();
    if (g.status) return;  // as StrokePass left it
    src.verbs = base + S.off[3];
    src.pts = (const P*)(base + S.off[4]);
    src.w = (const float*)(base + S.off[5]);
    src.nv = g.need[3];
    src.np = g.need[4];
    src.nw = g.need[5];
  } else {
    src = PassPath(b, pd);
  }
  const int k0 = stroke ? 9 : 0;
  DPath q;
  q.init(base + S.off[k0], pd.cap[k0], (P*)(base + S.off[k0 + 1]), pd.cap[k0 + 1],
         (float*)(base + S.off[k0 + 2]), pd.cap[k0 + 2]);
  QuadPathLanes(L, src, &q);
  g.need[k0] = q.nv;
  g.need[k0 + 1] = q.np;
  g.need[k0 + 2] = q.nw;
  if (q.overflow()) {
    g.status = 1;
    done();
    return;
  }
  const PathView quad = q.view();
  const Xform xf = PassXform(pd);
  const RasterBounds rb = pd.clipped ? BoundsLanes(L, quad, xf, pd.clip[0], pd.clip[1], pd.clip[2], pd.clip[3])
                                     : BoundsLanes(L, quad, xf, -1e9f, -1e9f, 1e9f, 1e9f);
  if (rb.empty) {
    done();
    return;
  }
  Edge* edges = (Edge*)(base + S.off[12]);
  const int n = BuildEdgesLanes(L, quad, xf, rb.st, rb.sb, edges, pd.cap[12]);
  g.need[12] = n;
  if (n > pd.cap[12] || n == 0) {
    g.status = n ? 1 : 0;
    done();
    return;
  }
  // sort the edges' keys, then the edges
  Edge* sorted = (Edge*)(base + S.off[13]);
  int32_t* idx = (int32_t*)(base + S.off[14]);
  SortKey* keys = n <= kSortKeys ? sh->keys : (SortKey*)sorted;
#pragma unroll 1
  for (int i = L.lane; i < n; i += NL) {
    SortKey k;
    k.y = edges[i].upper_y;
    k.x = edges[i].x;
    k.dx = edges[i].dx;
    k.idx = i;
    keys[i] = k;
  }
  L.sync();
  SortKeyLess less;
  IntrosortPartitions(L, sh, keys, n, less);
#pragma unroll 1
  for (int i = L.lane; i < n; i += NL) idx[StableRank(keys, n, i, less)] = keys[i].idx;
  L.sync();
  constexpr int kWords = (int)(sizeof(Edge) / 4);
#pragma unroll 1
  for (int t = L.lane; t < n * kWords; t += NL) {
    const int i = t / kWords;
    ((int32_t*)sorted)[t] = ((const int32_t*)(edges + idx[i]))[t - i * kWords];
  }
  L.sync();
  g.max_active = MaxActive(L, sh, sorted, n, (int32_t*)edges);

  const CanvasDesc cd = b.canvases[pd.canvas];
  g.n_edges = n;
  g.start_y = (int)rb.t;
  g.stop_y = (int)rb.sb;
  // static_cast<uint32_t>(float) << 16 with x86-64 conversion semantics
  g.left_bound = (Fixed)((uint32_t)(int64_t)rb.sl << 16);
  g.right_bound = (Fixed)((uint32_t)(int64_t)rb.sr << 16);
  g.acc_left = (int)rb.l;
  g.acc_width = (int)(rb.r - rb.l);
  g.scan_top = rb.st;
  // canvas rows; a ClipPath pass keeps all of its rows (the clip's span list
  // is empty or not over all rows, SWCanvas::State::HasClip)
  const bool all_rows = (pd.flags & kPassClipPath) != 0;
  const int r0 = all_rows ? g.start_y : max_(g.start_y, 0);
  const int r1 = all_rows ? g.stop_y : min_(g.stop_y, (int)cd.h);
  if (r0 < r1) {
    g.row0 = r0;
    g.row1 = r1;
  }
  done();
}

}  // namespace skc

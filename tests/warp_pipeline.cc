// Test-only: the pipeline as the GPU dispatches it, by 32 lanes a warp on the
// CPU (warp_lanes.h): geometry, each pass's sweep by the form its launch takes
// (SweepLaunch) with a warp that walks and a warp that emits, path clips by
// generation, the row tiles of BuildBalancedTasks.  cpu_pipeline.cc runs the
// same stages on one thread a pass.
#include "warp_lanes.h"

#include "../skity_gb300/csrc/batch.h"
#include "../skity_gb300/csrc/clip.cuh"
#include "../skity_gb300/csrc/passes.cuh"

using namespace skc;

static Lanes LaneOf(int lane) {
  Lanes L;
  L.lane = lane;
  return L;
}

// A pass by a pair of warps (k_sweep_pair); false: its list outgrew the form.
template <int M>
static bool Pair(const DevBatch& b, uint32_t p) {
  static RegPairT<M> sh;
  std::memset(&sh, 0x5A, sizeof sh);
  const int32_t cap = PairDiffCap<M>(b.reg_diff_cap);
  std::vector<int32_t> diff(cap, 0x5A5A);
  bool ok = true;
  lanes32::Run(2, [&](int warp, int lane) {
    const bool r = SweepPassPair<M, true>(b, p, LaneOf(lane), warp == 0, &sh, diff.data(), cap,
                                          [] { lanes32::MeetWarps(); });
    if (warp == 1 && lane == 0) ok = r;
  });
  return ok;
}

// The tiles cover every pixel of the canvases once and none is wider than the
// width returned, nor that than max_w.
static bool TilesCover(const HostBatch& hb, const std::vector<uint32_t>& canvases, uint32_t max_w,
                       std::vector<RowTask>& tasks) {
  const uint32_t widest = BuildBalancedTasks(hb, canvases, max_w, tasks);
  std::vector<std::vector<uint8_t>> seen(hb.canvases.size());
  uint64_t pixels = 0;
  for (uint32_t c : canvases) {
    seen[c].assign((size_t)hb.canvases[c].w * hb.canvases[c].h, 0);
    pixels += seen[c].size();
  }
  for (const RowTask& t : tasks) {
    if (t.x1 <= t.x0 || t.x1 - t.x0 > widest || t.canvas >= seen.size()) return false;
    const CanvasDesc& cd = hb.canvases[t.canvas];
    if (t.x1 > cd.w || t.y >= cd.h) return false;
    for (uint32_t x = t.x0; x < t.x1; ++x, --pixels)
      if (seen[t.canvas][(size_t)t.y * cd.w + x]++) return false;
  }
  return pixels == 0 && widest <= max_w;
}

// Every clip state with rows is in one generation, after its parent's.
static bool GenerationsHold(const HostBatch& hb, const std::vector<uint32_t>& order,
                            const std::vector<ClipGen>& gens) {
  std::vector<int> gen(hb.clip_states.size(), -1);
  uint32_t at = 0;
  for (size_t g = 0; g < gens.size(); ++g) {
    if (gens[g].first != at) return false;
    for (uint32_t i = 0; i < gens[g].count; ++i, ++at) {
      const ClipStateDesc& st = hb.clip_states[order[at] - 1];
      if (gen[order[at] - 1] >= 0 || (uint32_t)(st.y1 - st.y0) > gens[g].rows) return false;
      gen[order[at] - 1] = (int)g;
    }
  }
  for (size_t k = 0; k < gen.size(); ++k) {
    const ClipStateDesc& st = hb.clip_states[k];
    if ((gen[k] >= 0) != (st.y1 > st.y0)) return false;
    if (gen[k] >= 0 && st.parent && gen[st.parent - 1] >= gen[k]) return false;
  }
  return at == order.size();
}

// Renders a stream; forms: the passes each sweep form took (kSweepForms of
// them).  max_w: the widest tile; slack: edges taken off every pass's bound of
// its active list, so that it meets a form too small for it and is swept again.
extern "C" int skc_warp_render(const uint8_t* stream, size_t len, uint8_t* out, uint32_t max_w,
                               int slack, uint32_t* forms) {
  StreamView sv;
  if (!ParseStream(stream, len, &sv)) return -2;
  HostBatch hb;
  if (int rc = AddStreamCanvas(hb, sv)) return rc;
  const uint32_t np = (uint32_t)hb.passes.size();
  hb.verbs.push_back(0);
  hb.pts.push_back(mkP(0, 0));
  hb.weights.push_back(0);
  hb.stop_colors.push_back(make_float4(0, 0, 0, 0));
  hb.stop_offsets.push_back(0);
  hb.cf_matrices.push_back(0);
  std::vector<uint8_t> pixels(hb.pixel_bytes + 16, 0), roundtrip(256), srgb(512);
  for (const HostBatch::ImageUpload& u : hb.image_uploads)
    std::memcpy(pixels.data() + u.off, u.bytes.data(), u.bytes.size());
  for (int v = 0; v < 256; ++v) roundtrip[v] = ChannelToByte(v / 255.f);
  SRGBTables(srgb.data());

  std::vector<PassGeom> geom(np);
  std::vector<uint8_t> scratch;
  DevBatch b{};
  b.verbs = hb.verbs.data();
  b.pts = hb.pts.data();
  b.weights = hb.weights.data();
  b.draws = hb.draws.data();
  b.passes = hb.passes.data();
  b.n_passes = np;
  b.canvases = hb.canvases.data();
  b.geom = geom.data();
  b.brushes = hb.brushes.data();
  b.conicals = hb.conicals.data();
  b.srgb_tables = srgb.data();
  b.cf_matrices = hb.cf_matrices.data();
  b.stop_colors = hb.stop_colors.data();
  b.stop_offsets = hb.stop_offsets.data();
  b.pixels = pixels.data();
  b.roundtrip = roundtrip.data();
  for (bool again = true; again;) {
    uint64_t total = 0;
    for (PassDesc& pd : hb.passes) total = PlaceSlice(pd, total);
    scratch.assign(total + 16, 0);
    b.scratch = scratch.data();
    again = false;
    for (uint32_t p = 0; p < np; ++p) {
      static SortShared sort;
      lanes32::Run(1, [&](int, int lane) { StrokePass(b, p, LaneOf(lane)); });
      lanes32::Run(1, [&](int, int lane) { EdgesPass(b, p, LaneOf(lane), &sort); });
      if (!geom[p].status) continue;
      GrowCaps(hb.passes[p], geom[p]);
      again = true;
    }
  }
  for (PassGeom& g : geom) g.max_active = std::max(g.max_active - slack, 0);

  std::vector<PassSweep> sweep;
  const SweepPlan plan = PlanSweep(hb, geom, sweep);
  std::vector<uint8_t> sweepmem(plan.sweep_bytes + 16), pass_class(np + 1, 0);
  std::vector<uint2> rowspan(plan.rows + 1), pool(1024), clip_items;
  std::vector<uint32_t> pass_spans(np + 1), band_off, bins, order, clip_order;
  std::vector<PassComp> comp;
  PlanComp(hb, geom, sweep, comp);
  b.band_shift = 4;
  BuildBins(hb, comp, AssignBands(hb, b.band_shift), b.band_shift, band_off, bins);
  SweepOrder(geom, order);
  const uint64_t state_rows = PlanPathClips(hb, geom, clip_items);
  std::vector<ClipGen> gens;
  PlanClipGens(hb, clip_order, gens);
  if (!GenerationsHold(hb, clip_order, gens)) return -20;
  std::vector<uint32_t> clip_flags(2 * hb.clip_states.size() + 2);
  std::vector<uint2> clip_rows(state_rows + 1);
  std::vector<int32_t> clip_sort(kClipRowCap);
  uint32_t err = 0;
  unsigned long long next = 0;
  b.sweep = sweep.data();
  b.sweepmem = sweepmem.data();
  b.pass_class = pass_class.data();
  b.err = &err;
  b.rowspan = rowspan.data();
  b.pass_spans = pass_spans.data();
  b.comp = comp.data();
  b.band_off = band_off.data();
  b.bins = bins.data();
  b.reg_diff_cap = RegDiffCap(plan);
  b.clip_states = hb.clip_states.data();
  b.n_clip_states = (uint32_t)hb.clip_states.size();
  b.clip_flags = clip_flags.data();
  b.clip_rows = clip_rows.data();
  b.clip_items = clip_items.data();
  b.n_clip_items = (uint32_t)clip_items.size();
  b.span_next = &next;
  for (int attempt = 0;; ++attempt) {  // the pool grows until it holds everything
    if (attempt > 8 + (int)hb.clip_states.size()) return -7;
    next = 0;
    b.spans = pool.data();
    b.span_cap = pool.size();
    std::fill(rowspan.begin(), rowspan.end(), make_uint2(9, 9));
    std::fill(clip_flags.begin(), clip_flags.end(), 0u);
    std::fill(forms, forms + kSweepForms, 0u);
    std::vector<uint32_t> retry;
    for (uint32_t p : order) {
      const int form = SweepLaunch(geom[p], pass_class[p]);
      bool done = true;
      switch (form) {
        case kSweepReg32: done = Pair<32>(b, p); break;
        case kSweepReg64: done = Pair<64>(b, p); break;
        case kSweepReg128: done = Pair<128>(b, p); break;
        case kSweepReg256: done = Pair<256>(b, p); break;
        default: lanes32::Run(1, [&](int, int lane) { SweepPass(b, p, LaneOf(lane)); });
      }
      if (geom[p].n_edges > 0 && done) forms[form]++;
      if (!done) retry.push_back(p);
    }
    for (uint32_t p : retry) lanes32::Run(1, [&](int, int lane) { SweepPass(b, p, LaneOf(lane)); });
    for (uint32_t k : clip_order) {
      const ClipStateDesc& st = hb.clip_states[k - 1];
      for (int32_t y = st.y0; y < st.y1; ++y) ClipStateStage(b, k, y, clip_sort.data());
    }
    for (uint32_t i = 0; i < b.n_clip_items; ++i) ClipApplyStage(b, i, clip_sort.data());
    if (next <= pool.size()) break;
    pool.assign(2 * next, make_uint2(0, 0));
  }
  if (err) return -6;

  std::vector<uint32_t> row(65536);
  std::vector<RowTask> tasks;
  if (!TilesCover(hb, hb.temp_canvases, max_w, tasks)) return -21;
  for (const RowTask& t : tasks) CompositeRowScalar(b, t, row.data());
  for (uint32_t c : hb.temp_canvases)
    if (hb.canvases[c].blur_style != 0) return -22;  // layers only
  if (!TilesCover(hb, hb.main_canvases, max_w, tasks)) return -23;
  for (const RowTask& t : tasks) CompositeRowScalar(b, t, row.data());
  const CanvasDesc& cd = hb.canvases[hb.main_canvases[0]];
  std::memcpy(out, pixels.data() + cd.px_off, (size_t)cd.w * cd.h * 4);
  return 0;
}

// BuildBalancedTasks over canvases of the given sizes and passes.
extern "C" int skc_tiles_cover(int n, const uint32_t* w, const uint32_t* h, const uint32_t* passes,
                               uint32_t max_w) {
  HostBatch hb;
  std::vector<uint32_t> canvases;
  for (int i = 0; i < n; ++i) {
    CanvasDesc cd{};
    cd.w = w[i];
    cd.h = h[i];
    cd.pass1 = passes[i];
    canvases.push_back((uint32_t)hb.canvases.size());
    hb.canvases.push_back(cd);
  }
  std::vector<RowTask> tasks;
  return TilesCover(hb, canvases, max_w, tasks) ? 0 : 1;
}

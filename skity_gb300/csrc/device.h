// Device-side state of the raster pipeline shared by the batch / canvas C
// ABI (pipeline.cu) and the serving loop (server.cu): device buffers, a
// batch resident on the device, the context, and the pipeline entry points.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/skity_cuda.h"
#include "batch.h"

namespace skc {

// ---------------------------------------------------------------------------
// device buffers
// ---------------------------------------------------------------------------
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  ~DevBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap && p) return cudaSuccess;
    release();
    size_t want = std::max<size_t>(bytes, 256);
    cudaError_t e = cudaMalloc(&p, want);
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    cap = want;
    return cudaSuccess;
  }
  template <typename T>
  T* as() const { return (T*)p; }
};

// `v` to the start of `d`, grown to hold it.
template <typename T>
cudaError_t Upload(DevBuf& d, const std::vector<T>& v, cudaStream_t s) {
  cudaError_t e = d.ensure(std::max<size_t>(v.size() * sizeof(T), 16));
  if (e != cudaSuccess || v.empty()) return e;
  return cudaMemcpyAsync(d.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}

int32_t CudaErr(cudaError_t e);

struct Context;

// Launch shape of the compositor and the granularity of its pass bins
// (skity_cuda_raster_config; chosen per batch, e.g. by the autotuner).
struct RasterConfig {
  uint32_t tile_w = 1024;    // row-tile width in pixels
  uint32_t ctas_per_sm = 6;  // persistent compositor CTAs per SM (0: one warp per tile)
  int32_t band_shift = 4;    // pass-bin bands of 1 << band_shift rows
  uint32_t sweep_warps = 2;  // warps per CTA of the register sweeps (two a pass): 4, or 2 for 1 and 2
};

// A batch resident on the device: inputs uploaded once, re-rendered on
// demand.
struct DeviceBatch {
  Context* ctx = nullptr;
  HostBatch hb;
  DevBuf verbs, pts, weights, draws, passes, canvases, brushes, stop_colors, stop_offsets;
  DevBuf conicals, cf_matrices, srgb_tables;
  DevBuf scratch, geom, sweep, sweepmem, rowspan, pass_spans, comp, pixels;
  DevBuf tasks_main, tasks_temp, temps, pass_list, roundtrip, pass_frags, err, pass_class;
  DevBuf band_off, bins, sweep_order;
  std::vector<RowTask> h_tasks_main, h_tasks_temp;
  std::vector<uint32_t> h_band_off, h_bins;
  uint32_t chunk = 1024;
  uint32_t n_bands = 0;
  uint32_t any_stroke = 0;  // a pass is stroked
  RasterConfig cfg;
  DevBuf task_next;  // persistent compositor's counters
  DevBuf retry;      // DevBatch::sweep_retry
  DevBuf clip_states, clip_flags, clip_rows, clip_items, clip_order;  // path clips
  std::vector<ClipGen> clip_gens;
  // device planning (batches without path clips): status, per-pass scan
  // arrays and band ranges, bin segments, the tiles (main then temp) and
  // their sorted copy; capacities of the plan's buffers
  DevBuf plan_st, plan_a, plan_r, pband, segs, seg_cnt, tasks_in, tasks_sorted;
  DevBuf sort_keys, sort_hist;
  std::vector<BandSeg> h_segs;
  bool slices_dirty = true;   // pass capacities changed: slice offsets and passes re-uploaded
  uint64_t cap_sweep = 0, cap_rows = 0, cap_bins = 0;
  uint64_t slices_end = 0;    // end of the geometry slices in `scratch`
  // the launch parameters the replay graphs were recorded with
  DevBatch graph_b{};
  DevPlan graph_q{};
  int graph_launches = 0;
  // true when the caller has loaded the canvases' current pixels (a canvas
  // flush without a clear); otherwise a canvas without a clear colour starts
  // from transparent black, as a fresh Bitmap does
  bool keep_pixels = false;
  bool uploaded = false;
  // Replay of the planned render as one CUDA graph (device-resident
  // batches): the plan -- scratch capacities, sweep buffers, row tables,
  // bins -- depends only on the batch's inputs, so a re-render can run the
  // same launches on the same buffers without host round trips.
  bool want_graph = false;
  bool graph_ok = false;
  cudaGraphExec_t graphs[6] = {};
  DevBatch planned{};
  uint64_t planned_rows = 0;
  const void* planned_pool = nullptr;  // the context span pool the plan used
  skity_cuda_stats planned_stats{};
  ~DeviceBatch() {
    for (auto g : graphs)
      if (g) cudaGraphExecDestroy(g);
  }
  // Forgets the batch's canvases and draws but keeps its device buffers, so
  // the next batch built in it reuses their memory.
  void Reset() {
    for (auto& g : graphs) {
      if (g) cudaGraphExecDestroy(g);
      g = nullptr;
    }
    graph_ok = false;
    hb = HostBatch{};
    h_tasks_main.clear();
    h_tasks_temp.clear();
    h_band_off.clear();
    h_bins.clear();
    h_segs.clear();
    h_geom.clear();
    keep_pixels = false;
    uploaded = false;
    slices_dirty = true;
    slices_end = 0;
    cap_sweep = cap_rows = cap_bins = 0;
    stats = skity_cuda_stats{};
  }
  // Lays the passes' geometry slices out in `scratch`, one behind the other,
  // unless they stand, with room behind them for those that outgrow their
  // estimate.  Every renderer that keeps them for the next one does it here:
  // GrowSlices goes on where they end.
  int32_t LayoutSlices(uint64_t budget, cudaStream_t s) {
    if (!slices_dirty) return SKITY_CUDA_SUCCESS;
    uint64_t total = 0;
    for (PassDesc& pd : hb.passes) total = PlaceSlice(pd, total);
    if (budget && total > budget) return SKITY_CUDA_ERROR_OUT_OF_DEVICE_MEMORY;
    uint64_t want = total + total / 32 + (1u << 20);
    if (budget) want = std::max(total, std::min(want, budget));
    cudaError_t e = scratch.ensure(want);
    if (e == cudaSuccess) e = Upload(passes, hb.passes, s);
    if (e != cudaSuccess) return CudaErr(e);
    slices_dirty = false;
    slices_end = total;
    return SKITY_CUDA_SUCCESS;
  }
  // The passes whose geometry (h_geom) outgrew their slices get new ones
  // behind the others, and only they (`todo`) are to run again; without room
  // there, all slices are to be laid out again (slices_dirty).
  int32_t GrowSlices(std::vector<uint32_t>& todo, cudaStream_t s) {
    uint64_t end = slices_end;
    for (uint32_t p = 0; p < (uint32_t)hb.passes.size(); ++p) {
      if (!h_geom[p].status) continue;
      GrowCaps(hb.passes[p], h_geom[p]);
      end = PlaceSlice(hb.passes[p], end);
      todo.push_back(p);
    }
    slices_dirty = true;
    if (end > scratch.cap) return SKITY_CUDA_SUCCESS;
    if (cudaError_t e = Upload(passes, hb.passes, s)) return CudaErr(e);
    slices_dirty = false;
    slices_end = end;
    return SKITY_CUDA_SUCCESS;
  }
  std::vector<PassGeom> h_geom;
  skity_cuda_stats stats{};
};

}  // namespace skc

struct skity_cuda_context_s {
  int device = 0;
  uint64_t budget = 0;
  // span pool shared by the context's renders (they are serialised), grown
  // to what the largest render so far needed
  skc::DevBuf span_pool, span_next;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t stage[12] = {};
  // largest plan needs seen by the context's device-planned renders (sweep
  // bytes, row entries, bin entries): first capacities of new batches
  uint64_t hint_sweep = 0, hint_rows = 0, hint_bins = 0;
  // the batch skity_cuda_render_streams builds each call in (its device
  // buffers are reused from call to call)
  skc::DeviceBatch* streams_batch = nullptr;
  ~skity_cuda_context_s() { delete streams_batch; }
  skc::RasterConfig cfg;  // default launch shape of new batches and canvases
  uint32_t num_sms = 0;
  skity_cuda_stats last{};
  std::mutex mu;
};

namespace skc {

// Parses scene streams into the batch's host description.
int32_t BuildFromStreams(DeviceBatch& db, uint32_t count, const uint8_t* const* streams,
                         const size_t* bytes);
// Uploads the batch's inputs (once per batch).
int32_t UploadBatch(skity_cuda_context_s* ctx, DeviceBatch& db);
// Renders the batch on the context's stream (planned render, or the replay
// graphs when the batch has them); pixels stay on the device.
int32_t RenderBatch(skity_cuda_context_s* ctx, DeviceBatch& db, bool timed);
// Rebuilds the row tiles and bands of an uploaded batch for `cfg`; the next
// render plans again.
int32_t ApplyConfig(skity_cuda_context_s* ctx, DeviceBatch& db, const RasterConfig& cfg);
// Copies canvas `index` of the batch to host memory (row_bytes 0: packed).
int32_t ReadCanvas(skity_cuda_context_s* ctx, DeviceBatch& db, uint32_t index, uint8_t* out,
                   size_t row_bytes);
// Renders the batch's main canvases one DrawPath at a time (per_draw.cu);
// batches with blur mask filters or path clips are not taken.
int32_t RenderPerDraw(skity_cuda_context_s* ctx, DeviceBatch& db);
// Queues the copies of canvases [0, count) to out[i] (packed rows) on the
// context stream; the caller waits for the stream.
int32_t QueueReadCanvases(skity_cuda_context_s* ctx, DeviceBatch& db, uint32_t count,
                          uint8_t* const* out);

}  // namespace skc

// GB300 kernels of the raster pipeline.
//
//   k_stroke     1 warp / pass   : stroked passes: Path -> QuadPath -> outline
//   k_edges      1 warp / pass   : Path (or outline) -> QuadPath -> fixed-point
//                                  edges -> introsort
//   k_sweep_pair 2 warps / pass  : analytic-AA sweep, one walking, the other
//   k_sweep      1 warp / pass     one writing each row's spans contiguously
//                                  into the span pool; the generic form for
//                                  very long active lists
//   k_composite  1 warp / row tile: replays the spans of the row band's
//                                  passes in draw order into a shared-memory
//                                  tile, then writes the tile back
//   k_blur_h/_v  1 thread / channel of a row / column of each blur temp
//                                  canvas: StackBlur
//
// The stroker and the sweeps are inherently sequential per path (the
// reference's scanline sweep carries state across rows), so the parallelism
// there is across paths; compositing is parallel across rows and, inside a row,
// across the pixels of disjoint spans.
#include <cuda_runtime.h>

#include <algorithm>

#include "clip.cuh"
#include "overlap.cuh"
#include "passes.cuh"

namespace skc {

// Geometry, a warp a pass (edges.cuh): the stroker of the stroked passes, then
// quads, edges and sort.  With the whole chain on one thread, packed 1 to 32
// passes a warp, it was the batch's longest passes' serial chains, and half of
// a stroke's was double arithmetic (1/64 of the float rate).  Before / after:
// the 20,000-path scene 36.4 / 5.7 ms, 64 canvases of fills 3.3 / 0.84, a
// picture of 305 long outlines 32.7 / 4.6, 512x512 of 1,000 fills 0.70 / 0.09.
// (k_edges overlapping k_stroke, stroked passes alone waiting for it, is
// slower: 6.3 ms for the scene, and 2.58 instead of 2.13 for 110,000 glyphs.)
constexpr int kGeomWarps = 4;
__global__ void __launch_bounds__(32 * kGeomWarps) k_stroke(DevBatch b) {
  const uint32_t i = blockIdx.x * kGeomWarps + (threadIdx.x >> 5);
  if (i >= b.n_list) return;
  Lanes L;
  L.lane = threadIdx.x & 31;
  StrokePass(b, b.pass_list ? b.pass_list[i] : i, L);
}

__global__ void __launch_bounds__(32 * kGeomWarps) k_edges(DevBatch b) {
  __shared__ SortShared sh[kGeomWarps];
  const uint32_t i = blockIdx.x * kGeomWarps + (threadIdx.x >> 5);
  if (i >= b.n_list) return;
  Lanes L;
  L.lane = threadIdx.x & 31;
  EdgesPass(b, b.pass_list ? b.pass_list[i] : i, L, &sh[threadIdx.x >> 5]);
}

int LaunchGeometry(const DevBatch& b, cudaStream_t stream) {
  if (b.n_list == 0) return 0;
  const uint32_t grid = (b.n_list + kGeomWarps - 1) / kGeomWarps;
  int n = 1;
  if (b.any_stroke) {
    k_stroke<<<grid, 32 * kGeomWarps, 0, stream>>>(b);
    n++;
  }
  k_edges<<<grid, 32 * kGeomWarps, 0, stream>>>(b);
  return n;
}

// Sweeps, passes taken in the batch's sweep order
// (longest expected sweeps first, so the long ones do not form the tail).
// Five forms, each taking the passes SweepLaunch gives it: register forms for
// up to 32, 64, 128 and 256 active edges (two warps a pass, its RegPairT block
// and accumulator in shared memory), then the generic sweep (4 warps per
// block, state in global memory) for longer lists.
constexpr int kSweepWarps = 4;

__device__ __forceinline__ uint32_t DynamicSmemBytes() {
  uint32_t v;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(v));
  return v;
}

// The i-th pass of a sweep form (n_passes: there is none).  A device plan
// lists each form's passes together, and a plan that fell short sweeps
// nothing (the host renders again with its buffers grown); without a plan the
// form's launch goes through all passes.
__device__ __forceinline__ uint32_t SweepPassAt(const DevBatch& b, int form, uint32_t i) {
  if (b.plan) {
    const uint32_t at = b.plan->form_end[form + 1] + i;
    return (b.plan->flags || at >= b.plan->form_end[form]) ? b.n_passes : b.sweep_order[at];
  }
  if (i >= b.n_passes) return b.n_passes;
  const uint32_t p = b.sweep_order ? b.sweep_order[i] : i;
  return SweepLaunch(b.geom[p], b.pass_class[p]) == form ? p : b.n_passes;
}

// End of a sweep kernel that may have overlapped the one before it: the
// CTA that finishes last waits for that kernel to complete, so this kernel
// completes only after every earlier sweep kernel has, and the work queued
// after the sweeps sees all of them done.  (In a launch that overlapped
// nothing the wait returns at once.)
__device__ __forceinline__ void FinishOverlapped(unsigned int* done) {
  if (!done) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(done, 1u) == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
  }
}

// Waits for the other warp of the pair (at most two pairs per CTA; literal
// barrier numbers, a CTA holds on to as many as its code may name).
__device__ __forceinline__ void MeetPair(int pair) {
  if (pair == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
  else asm volatile("bar.sync 2, 64;" ::: "memory");
}

// Pairs per SM that the registers leave room for.  More pairs hide
// more latency until the compiler runs out of registers for the walk: of the
// 32-edge form 11 fit without a cap; 12 / 13 / 15 pairs sweep 64 canvases of
// 50-2,000 paths in 14.3 / 14.0 / 14.1 ms (11: 15.6), 1,000 paths on 512 x
// 512, where latency counts, in 1.99 / 2.08 / 2.18 (11: 1.97).
template <int M>
constexpr int kPairsPerSm = M == 32 ? 12 : M == 64 ? 10 : 2;

// A pass is swept by two warps: one walks the active list and logs intervals,
// the other one makes the spans of the log before (SweepPassPair).
//
// What bounds it: a pass is a chain of quarter-pixel steps, one after the
// other, some 2 us each when one warp both walks and emits; large batches are
// bound by instruction issue.  With a step's coverage made inside the step,
// the kernel was 140 KB of unrolled code, and instruction fetch held it at
// 26-34 % of the issue slots; walk and emission as two short loops
// (regsweep.cuh), one copy of each part and no unrolling are 54 KB and issue
// 53 %, with fewer instructions a span (105 -> 73): 64 canvases of 50-2,000
// paths 38 -> 15.5 ms.  The loops on two warps instead of in turns on one:
// half the chain, and 80 registers instead of 124, so nearly as many passes
// are in flight.  1,000 paths on 512 x 512 2.71 -> 1.91 ms, 305 long strokes
// and fills 12.8 -> 8.2, 400 effects draws 2.70 -> 1.99, the 64 canvases
// 15.5 -> 13.9, 110,000 glyphs 8.4 -> 7.0; 20,000 paths of 64 verbs, most in
// the 64-edge form, 154 -> 157.
template <int M, int kForm, bool kRaw>
__global__ void __launch_bounds__(128, kPairsPerSm<M> / 2) k_sweep_pair(DevBatch b) {
  extern __shared__ __align__(16) uint8_t reg_smem[];
  AllowNextLaunch();
  const int pair = threadIdx.x >> 6;
  const uint32_t pairs = blockDim.x >> 6;
  const uint32_t p = SweepPassAt(b, kForm, blockIdx.x * pairs + pair);
  if (p < b.n_passes) {  // the same for both warps
    const int32_t diff_cap = PairDiffCap<M>(b.reg_diff_cap);
    if (DynamicSmemBytes() < pairs * PairSmemBytes<M>(diff_cap)) {  // self-check
      FlagError(b.err, 16);
    } else {
      Lanes L;
      L.lane = threadIdx.x & 31;
      uint8_t* mine = reg_smem + (size_t)pair * PairSmemBytes<M>(diff_cap);
      if (!SweepPassPair<M, kRaw>(b, p, L, (threadIdx.x & 32) == 0, (RegPairT<M>*)mine,
                                  (int32_t*)(mine + sizeof(RegPairT<M>)), diff_cap,
                                  [pair] { MeetPair(pair); }) &&
          L.leader()) {
        // each pass is taken by one form, so the list holds at most n_passes
        const uint32_t at = b.sweep_retry ? atomicAdd(b.sweep_retry, 1u) : b.n_passes;
        if (at < b.n_passes) {
          b.sweep_retry[1 + at] = p;
        } else {
          FlagError(b.err, 32);  // no list: the pass stays unswept, the render fails
        }
      }
    }
  }
  FinishOverlapped(b.sweep_done ? b.sweep_done + kForm : nullptr);
}

// The passes the register forms gave up on, swept with the generic form after
// every register form has finished (a plain launch after them).  The last CTA
// marks the plan of a render whose sweeps ran out of span pool: the compositor
// then has one word to look at (reading the pool's counter there changed its
// register allocation: 1,500 paths with gradients 3.72 -> 3.82 ms).
__global__ void __launch_bounds__(32 * kSweepWarps) k_sweep_retry(DevBatch b) {
  if (!b.sweep_retry) return;
  const uint32_t n = min(b.sweep_retry[0], b.n_passes);
  const uint32_t nw = gridDim.x * kSweepWarps;
  Lanes L;
  L.lane = threadIdx.x & 31;
  for (uint32_t i = blockIdx.x * kSweepWarps + (threadIdx.x >> 5); i < n; i += nw)
    SweepPass(b, b.sweep_retry[1 + i], L);
  if (!b.plan) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(b.sweep_done + kSweepForms, 1u) == gridDim.x - 1 &&
        *(volatile unsigned long long*)b.span_next > b.span_cap)
      atomicOr(&b.plan->flags, (uint32_t)kPlanSpans);
  }
}

template <bool kRaw>
__global__ void __launch_bounds__(32 * kSweepWarps) k_sweep(DevBatch b) {
  AllowNextLaunch();
  const uint32_t p =
      SweepPassAt(b, kSweepGeneric, blockIdx.x * kSweepWarps + (threadIdx.x >> 5));
  if (p < b.n_passes) {
    Lanes L;
    L.lane = threadIdx.x & 31;
    SweepPass<kRaw>(b, p, L);
  }
  FinishOverlapped(b.sweep_done ? b.sweep_done + kSweepGeneric : nullptr);
}

template <int M, int kForm, bool kRaw>
static void LaunchRegForm(const DevBatch& b, cudaStream_t stream, bool overlap) {
  const uint32_t pairs = b.reg_warps == 4 ? 2 : 1;
  const size_t smem = pairs * PairSmemBytes<M>(PairDiffCap<M>(b.reg_diff_cap));
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(k_sweep_pair<M, kForm, kRaw>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
  LaunchOverlapped(k_sweep_pair<M, kForm, kRaw>, dim3((b.n_passes + pairs - 1) / pairs),
                   dim3(64 * pairs), smem, stream, overlap, b);
}

// The sweep forms in launch order: heaviest first, so the longest sweeps start
// at once and each later (lighter) form fills the SMs the earlier ones' tails
// leave idle.  They may overlap: they take disjoint passes and read nothing
// the others write.  kRaw: the batch has path clips, whose passes keep raw
// spans.
template <bool kRaw>
static void LaunchForms(const DevBatch& b, cudaStream_t stream, bool overlap) {
  LaunchOverlapped(k_sweep<kRaw>, dim3((b.n_passes + kSweepWarps - 1) / kSweepWarps),
                   dim3(32 * kSweepWarps), 0, stream, false, b);
  LaunchRegForm<256, kSweepReg256, kRaw>(b, stream, overlap);
  LaunchRegForm<kRegMaxM, kSweepReg128, kRaw>(b, stream, overlap);
  LaunchRegForm<64, kSweepReg64, kRaw>(b, stream, overlap);
  LaunchRegForm<32, kSweepReg32, kRaw>(b, stream, overlap);
}

// With b.sweep_done (a zeroed counter per form) the later forms overlap the
// earlier ones' tails; without, they run one after the other.
int LaunchSweep(const DevBatch& b, cudaStream_t stream) {
  if (b.n_passes == 0) return 0;
  const bool overlap = b.sweep_done != nullptr;
  if (b.n_clip_states)
    LaunchForms<true>(b, stream, overlap);
  else
    LaunchForms<false>(b, stream, overlap);
  k_sweep_retry<<<64, 32 * kSweepWarps, 0, stream>>>(b);
  return kSweepForms + 1;
}

// ---------------------------------------------------------------------------
// composite: one warp per row tile (x0, x1) of a canvas row, the tile held in
// shared memory.  The passes come from the row band's bin (draw order); each
// pass row's spans are loaded 32 at a time, the ones meeting the tile are
// applied in emission order, in batches of disjoint spans (every pixel's
// blends stay in the reference's order).  A batch's pixels are numbered
// through its spans and taken 32 at a time, whatever their spans' lengths, so
// the lanes stay full: a lane finds its pixel's span from a bit mask of the
// span starts among the 32.  (With short spans on a lane each and long ones
// by the whole warp in turn, 3.45 warp instructions a solid fragment.)
// ---------------------------------------------------------------------------
constexpr int kCompWarps = 4;
// CTAs per SM the compositor's register budget leaves room for (its stalls
// are mostly dependent integer chains: more resident warps hide them)
constexpr int kCompMinBlocks = 6;

// gradient stops a warp stages in shared memory (longer gradients are read
// from global memory)
constexpr int kStagedStops = 16;
// shared memory of one compositor warp: its tile row, padded to 16 bytes (a
// tile may be any number of pixels wide, the stop colours are read as
// float4), then the staged stops (colours, offsets, reciprocals, cells), then
// a batch's spans (two words each)
__host__ __device__ constexpr size_t CompRowBytes(uint32_t chunk) {
  return ((size_t)chunk * 4 + 15) & ~(size_t)15;
}
__host__ __device__ constexpr size_t CompWarpSmem(uint32_t chunk) {
  return CompRowBytes(chunk) + kStagedStops * (16 + 4 + 4) + 32 + 32 * 8;
}
struct CompShared {  // the parts of a warp's shared memory
  uint32_t* row;
  StagedStops stops;
  uint2* spans;
};

template <bool kAll>
__device__ __forceinline__ void CompositeTile(const DevBatch& b, const RowTask& rt,
                                              const CompShared& sh, int lane);

// counter == null: warp w of block k takes tile 4k + w; otherwise every warp
// takes tiles from the counter until none is left (persistent grid).
// kAll: the general form (every brush kind, colour filter and blend mode),
// launched for batches with a general canvas; the common form has no calls
// and keeps its loops in registers.
template <bool kAll>
__global__ void __launch_bounds__(32 * kCompWarps, kCompMinBlocks)
    k_composite(DevBatch b, const RowTask* __restrict__ tasks, uint32_t n_tasks, uint32_t chunk,
                unsigned int* counter) {
  extern __shared__ __align__(16) uint8_t reg_smem[];
  // a device plan that fell short, or sweeps that ran out of span pool: the
  // host grows the buffers and renders again, so nothing is composited (a
  // canvas that keeps its pixels would get the spans there are twice)
  if (b.plan && b.plan->flags) return;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  uint8_t* mine = reg_smem + (size_t)wib * CompWarpSmem(chunk);
  CompShared sh;
  sh.row = (uint32_t*)mine;
  sh.stops.colors = (float4*)(mine + CompRowBytes(chunk));
  sh.stops.offsets = (float*)(sh.stops.colors + kStagedStops);
  sh.stops.recip = sh.stops.offsets + kStagedStops;
  sh.stops.first = (uint8_t*)(sh.stops.recip + kStagedStops);
  sh.spans = (uint2*)(sh.stops.first + 32);
  if (!counter) {
    const uint32_t task = blockIdx.x * kCompWarps + wib;
    if (task < n_tasks) CompositeTile<kAll>(b, tasks[task], sh, lane);
    return;
  }
  for (;;) {
    uint32_t task = 0;
    if (lane == 0) task = atomicAdd(counter, 1u);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= n_tasks) return;
    CompositeTile<kAll>(b, tasks[task], sh, lane);
    __syncwarp();
  }
}

// The head of a brush: what solid fills need.
struct BrushHead {
  uint32_t kind, blend, solid, global_alpha;
};

// The spans of a pass row are one dependent load behind its row entry; those
// of 32 passes start on their way to the L2 at once (64 canvases of 50-2,000
// paths: 3.52 -> 3.28 ms; spans in registers two passes ahead instead: 3.56).
__device__ __forceinline__ void PrefetchL2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// How a pass's pixels are made.
//   solid:    a src-over fill without a colour filter: the span's colour is
//             made once a span, and a pixel is one PMSrcOver.  FastBlend's
//             shortcuts need no test: premultiplied colours of alpha 0 are 0,
//             and 256 - alpha is 1 for alpha 255, which leaves nothing of the
//             destination.
//   gradient: a linear or radial one, src-over, no colour filter, whose stops
//             GradientColorStaged takes; blended the same way.
//   other:    everything else, pixel by pixel as the reference does it.
enum CompKind { kCompSolid, kCompGradient, kCompOther };

// The spans [s0, s1) of one pass row applied to the row tile; `mine`: this
// lane's span of the first 32, already loaded.
template <bool kAll, int kKind>
__device__ __forceinline__ void CompositeSpans(const DevBatch& b, const BrushHead& bh,
                                               const Brush& br, const CompShared& sh, uint2 mine,
                                               uint32_t s0, uint32_t s1, int x0, int x1, int y,
                                               int lane) {
  uint32_t* row = sh.row;
  const uint32_t le = (2u << lane) - 1u;
  const float4* stop_colors = b.stop_colors;
  const float* stop_offsets = b.stop_offsets;
  // one pixel; v: the span's colour (solid) or alpha
  auto pixel = [&](int px, uint32_t v) {
    uint32_t& d = row[px];
    if (kKind == kCompSolid) {
      d = PMSrcOver(v, d);
    } else if (kKind == kCompGradient) {
      const float sx = (px + x0) + 0.5f, sy = y + 0.5f;
      const float mx = sx * br.m[0] + sy * br.m[1] + br.m[2];
      float t = mx;
      if (br.kind == 2) {
        const float my = sx * br.m[3] + sy * br.m[4] + br.m[5];
        t = sqrt_(mx * mx + my * my);
      }
      uint32_t c = GradientColorStaged(br.tile, (int)br.stop_count, t, sh.stops);
      if (v != 255) c = AlphaMulQ(c, v);
      d = PMSrcOver(c, d);
    } else {
      uint32_t c = kAll ? BrushColor(br, px + x0, y, stop_colors, stop_offsets, b.pixels,
                                     b.roundtrip, b.conicals)
                        : BrushColorCommon(br, px + x0, y, stop_colors, stop_offsets, b.pixels,
                                           b.roundtrip);
      if (v != 255) c = AlphaMulQ(c, v);
      if (kAll && br.cf_type) c = FilterColor(br, c, b.srgb_tables, b.cf_matrices);
      d = kAll ? BlendPixel(d, c, br.blend) : BlendPixelCommon(d, c, br.blend);
    }
  };
#pragma unroll 1
  for (uint32_t sb = s0; sb < s1; sb += 32) {
    int xs = 0, xe = 0;
    uint32_t v = 0;
    if (sb + lane < s1) {
      xs = max((int)(mine.x & 0xFFFF), x0);
      xe = min((int)(mine.x & 0xFFFF) + (int)(mine.x >> 16), x1);
      v = mine.y & bh.global_alpha;
      if (kKind == kCompSolid) v = v != 255 ? AlphaMulQ(bh.solid, v) : bh.solid;
    }
    if (sb + 32 + lane < s1) mine = b.spans[sb + 32 + lane];
    // Spans are applied in batches: the longest run of pending spans (in
    // emission order) in which each starts at or after the end of the one
    // before.  Those are disjoint, so inside a batch the order does not
    // matter.
    uint32_t pmask = __ballot_sync(0xffffffffu, xs < xe);
#pragma unroll 1
    while (pmask) {
      const bool pending = (pmask >> lane) & 1u;
      const uint32_t below = pmask & (le >> 1);
      const int prev_xe = __shfl_sync(0xffffffffu, xe, below ? 31 - __clz(below) : lane);
      const uint32_t cmask = __ballot_sync(0xffffffffu, pending && below && prev_xe > xs);
      const uint32_t batch = cmask ? pmask & ((1u << (__ffs(cmask) - 1)) - 1u) : pmask;
      const bool now = (batch >> lane) & 1u;
      int len = now ? xe - xs : 0;
      int at = xs - x0;
      // whole blocks of 32 pixels of the long spans, a lane a pixel
      if (kKind != kCompOther) {
        uint32_t lmask = __ballot_sync(0xffffffffu, len >= 32);
#pragma unroll 1
        while (lmask) {
          const int j = __ffs(lmask) - 1;
          lmask &= lmask - 1;
          const int q = __shfl_sync(0xffffffffu, at, j) + lane;
          const int n = __shfl_sync(0xffffffffu, len, j) & ~31;
          const uint32_t qv = __shfl_sync(0xffffffffu, v, j);
#pragma unroll 1
          for (int i = 0; i < n; i += 32) pixel(q + i, qv);
        }
        at += len & ~31;
        len &= 31;
        __syncwarp();
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      const int excl = incl - len;
      // the pixels left over, numbered through the batch's spans (packed:
      // pixel - number, colour or alpha) and taken 32 at a time
      const uint32_t some = kKind != kCompOther ? __ballot_sync(0xffffffffu, len > 0) : batch;
      if ((some >> lane) & 1u)
        sh.spans[__popc(some & (le >> 1))] = make_uint2((uint32_t)(at - excl), v);
      __syncwarp();
      int before = -1;  // spans that start before the 32 pixels, less one
#pragma unroll 1
      for (int w = 0; w < total; w += 32) {
        const uint32_t rel = (uint32_t)(excl - w);
        const uint32_t starts =
            __reduce_or_sync(0xffffffffu, (len > 0 && rel < 32u) ? 1u << rel : 0u);
        const int g = w + lane;
        if (g < total) {
          const uint2 sp = sh.spans[before + __popc(starts & le)];
          pixel((int)sp.x + g, sp.y);
        }
        before += __popc(starts);
      }
      __syncwarp();
      pmask &= ~batch;
    }
  }
}

// Stages a gradient's stops for a warp; whether GradientColorStaged takes it.
__device__ __forceinline__ bool StageStops(const DevBatch& b, const Brush& br,
                                           const StagedStops& st, int lane) {
  const int n = (int)br.stop_count;
  if (n < 2 || n > kStagedStops || !br.has_offsets) return false;
  float4 c = make_float4(0, 0, 0, 0);
  float o = 0;
  if (lane < n) {
    c = b.stop_colors[br.stop0 + lane];
    o = b.stop_offsets[br.stop0 + lane];
  }
  const float next = __shfl_down_sync(0xffffffffu, o, 1);
  const bool fits = lane >= n || StagedStop(c, o, lane < n - 1 ? next : o);
  if (!__all_sync(0xffffffffu, fits)) return false;
  __syncwarp();
  if (lane < n) {
    st.colors[lane] = c;
    st.offsets[lane] = o;
    st.recip[lane] = 1.0f / (next - o);
  }
  __syncwarp();
  st.first[lane] = (uint8_t)FirstInterval(st.offsets, n, lane);
  __syncwarp();
  return true;
}

template <bool kAll>
__device__ __forceinline__ void CompositeTile(const DevBatch& b, const RowTask& rt,
                                              const CompShared& sh, int lane) {
  const CanvasDesc cd = b.canvases[rt.canvas];
  const int y = (int)rt.y;
  const int x0 = (int)rt.x0, x1 = (int)rt.x1;
  const int n = x1 - x0;
  uint32_t* row = sh.row;
  uint32_t* gpx = (uint32_t*)(b.pixels + cd.px_off) + (size_t)y * cd.w + x0;
#pragma unroll 1
  for (int i = lane; i < n; i += 32) {
    row[i] = cd.has_clear ? cd.clear_pm : RGBAtoARGB(gpx[i]);
  }
  __syncwarp();
  const uint32_t band = cd.band0 + ((uint32_t)y >> b.band_shift);
  const uint32_t e0 = b.band_off[band], e1 = b.band_off[band + 1];
  // 32 bin entries at a time: each lane looks up its pass's row entry and
  // brush, so the loads of 32 passes are in flight together and passes with
  // no spans on this row cost no serial step
#pragma unroll 1
  for (uint32_t eb = e0; eb < e1; eb += 32) {
    const uint32_t e = eb + lane;
    uint2 rs = make_uint2(0, 0);
    uint32_t brush = 0;
    if (e < e1) {
      const PassComp pc = b.comp[b.bins[e]];
      if (y >= pc.row0 && y < pc.row1) {
        rs = b.rowspan[pc.rbase + (y - pc.row0)];
        brush = pc.brush;
      }
    }
    BrushHead bh = {0, 0, 0, 0};
    if (rs.y != 0) {
      const Brush& q = b.brushes[brush];
      bh.kind = q.kind;
      bh.blend = q.blend;
      bh.solid = q.solid;
      bh.global_alpha = q.global_alpha;
    }
    if (rs.y != 0) PrefetchL2(b.spans + rs.x);
    if (rs.y > 16) PrefetchL2(b.spans + rs.x + 16);
    uint32_t mask = __ballot_sync(0xffffffffu, rs.y != 0);
    // the first 32 spans of a pass are loaded while the pass before is blended
    auto first_spans = [&](uint32_t m) {
      const int bit = m ? __ffs(m) - 1 : 0;
      const uint32_t f0 = __shfl_sync(0xffffffffu, rs.x, bit);
      const uint32_t fn = __shfl_sync(0xffffffffu, rs.y, bit);
      uint2 v = make_uint2(0, 0);
      if (m && lane < (int)min(fn, 32u)) v = b.spans[f0 + lane];
      return v;
    };
    uint2 next = first_spans(mask);
#pragma unroll 1
    while (mask) {
      const int bit = __ffs(mask) - 1;
      mask &= mask - 1;
      const uint2 mine = next;
      next = first_spans(mask);
      const uint32_t s0 = __shfl_sync(0xffffffffu, rs.x, bit);
      const uint32_t s1 = s0 + __shfl_sync(0xffffffffu, rs.y, bit);
      const uint32_t qbrush = __shfl_sync(0xffffffffu, brush, bit);
      BrushHead qh;
      qh.kind = __shfl_sync(0xffffffffu, bh.kind, bit);
      qh.blend = __shfl_sync(0xffffffffu, bh.blend, bit);
      qh.solid = __shfl_sync(0xffffffffu, bh.solid, bit);
      qh.global_alpha = __shfl_sync(0xffffffffu, bh.global_alpha, bit);
      Brush br;
      if (qh.kind == 0 && qh.blend == 3 && (!kAll || b.brushes[qbrush].cf_type == 0)) {
        CompositeSpans<kAll, kCompSolid>(b, qh, br, sh, mine, s0, s1, x0, x1, y, lane);
        continue;
      }
      br = b.brushes[qbrush];
      if ((qh.kind == 1 || qh.kind == 2) && qh.blend == 3 && (!kAll || br.cf_type == 0) &&
          StageStops(b, br, sh.stops, lane))
        CompositeSpans<kAll, kCompGradient>(b, qh, br, sh, mine, s0, s1, x0, x1, y, lane);
      else
        CompositeSpans<kAll, kCompOther>(b, qh, br, sh, mine, s0, s1, x0, x1, y, lane);
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < n; i += 32) gpx[i] = ARGBtoRGBA(row[i]);
}

int LaunchComposite(const DevBatch& b, const RowTask* tasks, uint32_t n_tasks, uint32_t chunk,
                    uint32_t ctas_per_sm, uint32_t num_sms, unsigned int* counter,
                    cudaStream_t stream) {
  if (n_tasks == 0) return 0;
  size_t smem = (size_t)kCompWarps * CompWarpSmem(chunk);
  auto kernel = b.any_general ? k_composite<true> : k_composite<false>;
  if (smem > 48 * 1024) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }
  uint32_t grid = (n_tasks + kCompWarps - 1) / kCompWarps;
  if (ctas_per_sm > 0 && counter) {
    grid = std::min<uint32_t>(grid, ctas_per_sm * std::max<uint32_t>(num_sms, 1));
  } else {
    counter = nullptr;
  }
  kernel<<<grid, 32 * kCompWarps, smem, stream>>>(b, tasks, n_tasks, chunk, counter);
  return 1;
}

// ---------------------------------------------------------------------------
// Path clips (clip.cuh): the clip states' span rows, a thread a row, one
// launch per generation (a state reads its parent's rows and whether the
// parent's list is empty, known only once the parent's launch is complete;
// with a launch per state, 24 states in groups of three took 0.4 ms longer),
// then the rows of the draws under a clip, one thread per (pass, row).
// ---------------------------------------------------------------------------
constexpr int kClipThreads = 128;
__global__ void __launch_bounds__(kClipThreads) k_clip_state(DevBatch b, const uint32_t* states) {
  const uint32_t k = states[blockIdx.y];
  const ClipStateDesc& st = b.clip_states[k - 1];
  const int32_t y = st.y0 + (int32_t)(blockIdx.x * kClipThreads + threadIdx.x);
  if (y >= st.y1) return;
  int32_t order[kClipRowCap];
  ClipStateStage(b, k, y, order);
}

__global__ void __launch_bounds__(kClipThreads) k_clip_apply(DevBatch b) {
  const uint32_t i = blockIdx.x * kClipThreads + threadIdx.x;
  if (i >= b.n_clip_items) return;
  int32_t order[kClipRowCap];
  ClipApplyStage(b, i, order);
}

int LaunchPathClips(const DevBatch& b, const uint32_t* order, const ClipGen* gens, size_t n_gens,
                    cudaStream_t stream) {
  int launches = 0;
  for (size_t g = 0; g < n_gens; ++g) {
    for (uint32_t at = 0; at < gens[g].count; at += 65535) {
      const dim3 grid((gens[g].rows + kClipThreads - 1) / kClipThreads,
                      std::min(gens[g].count - at, 65535u));
      k_clip_state<<<grid, kClipThreads, 0, stream>>>(b, order + gens[g].first + at);
      launches++;
    }
  }
  if (b.n_clip_items) {
    k_clip_apply<<<(b.n_clip_items + kClipThreads - 1) / kClipThreads, kClipThreads, 0, stream>>>(b);
    launches++;
  }
  return launches;
}

// ---------------------------------------------------------------------------
// StackBlur (src/render/sw/sw_stack_blur.cc:18-284) on blur temp canvases.
// The reference's ring buffer only ever holds input pixels at clamped
// indices, so each step reads them directly: the value leaving the left half
// is pixel(max(i - r, 0)), the one entering is pixel(min(i + r + 1, n - 1)),
// the one crossing the centre is pixel(min(i + 1, n - 1)).  Horizontal pass:
// canvas -> blur scratch; vertical pass: blur scratch -> canvas.
// ---------------------------------------------------------------------------
// A thread blurs one channel of one line.  What bounds it is the running sum's
// chain along the line: a thread a line, four channels in 64-bit sums, took
// four times as long a step, and the small blurs of a page (15 to 80 pixels)
// are a few lines long: 8 blurs of a page 0.170 -> 0.035 ms, 10,000 glyph blurs
// 1.38 -> 0.55.
//
// Staged StackBlur: a block copies a run of whole rows (horizontal pass) or
// a 32-column strip of every row (vertical pass) of one temp canvas into
// shared memory with coalesced 4-byte loads -- the rows are contiguous in
// memory, and 32 lanes cover 128 contiguous bytes of a strip row.  The
// horizontal pass blurs into shared memory too and writes the rows back
// coalesced, the vertical one into global memory (the threads are on the same
// row at a time).  Lines are stored an odd number of words apart, so the
// threads, each walking its own line, hit distinct banks.  Temp canvases whose
// lines do not fit the shared-memory budget take the direct kernels (they
// return at once for the staged ones, and the staged ones for them).
constexpr int kBlurRows = 64;     // rows of a horizontal block, at most
constexpr int kBlurThreads = 4 * kBlurRows;
constexpr int kBlurStrip = 32;    // columns of a vertical block
constexpr int kBlurStripThreads = 4 * kBlurStrip;
constexpr uint32_t kBlurSmemWords = 12 * 1024;  // 48 KiB: input (and output) lines

__host__ __device__ inline uint32_t OddStride(uint32_t n) { return n | 1u; }
// Rows per block of the staged horizontal pass (0: the row does not fit).
__host__ __device__ inline uint32_t BlurRowsPerBlock(uint32_t w) {
  const uint32_t r = kBlurSmemWords / (2 * OddStride(w));
  return r < (uint32_t)kBlurRows ? r : (uint32_t)kBlurRows;
}
// The staged vertical pass takes canvases whose strip fits.
__host__ __device__ inline bool BlurStripFits(uint32_t h) {
  return (uint64_t)OddStride(kBlurStrip) * h <= kBlurSmemWords;
}

// Channel c of a line of n pixels, `step` bytes apart (`out_step` in the
// output), blurred, or copied (a blur of radius 1).  v: the vertical pass.
__device__ __forceinline__ void BlurOrCopy(const uint8_t* line, size_t step, uint8_t* out,
                                           size_t out_step, int n, int radius, int c, bool v) {
  const int r = min(radius, 254);
  if (r <= 1) {
    for (int i = 0; i < n; ++i) out[c + (size_t)i * out_step] = line[c + (size_t)i * step];
    return;
  }
  BlurChannel(line + c, step, out + c, out_step, n, r, line[v && (c == 0 || c == 3) ? 1 : c]);
}

__global__ void k_blur_h(DevBatch b, const uint32_t* temps, uint32_t n_temp) {
  const uint32_t t = blockIdx.y;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, y = i >> 2;
  if (t >= n_temp) return;
  const CanvasDesc cd = b.canvases[temps[t]];
  // staged, or a layer's temp canvas (no blur)
  if (y >= cd.h || BlurRowsPerBlock(cd.w) != 0 || cd.blur_style == 0) return;
  BlurOrCopy(b.pixels + cd.px_off + (size_t)y * cd.w * 4, 4,
             b.pixels + cd.blur_off + (size_t)y * cd.w * 4, 4, (int)cd.w, cd.blur_radius, i & 3,
             false);
}

__global__ void k_blur_v(DevBatch b, const uint32_t* temps, uint32_t n_temp) {
  const uint32_t t = blockIdx.y;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, x = i >> 2;
  if (t >= n_temp) return;
  const CanvasDesc cd = b.canvases[temps[t]];
  if (x >= cd.w || BlurStripFits(cd.h) || cd.blur_style == 0) return;  // staged, or a layer
  const size_t step = 4 * (size_t)cd.w;
  BlurOrCopy(b.pixels + cd.blur_off + (size_t)x * 4, step, b.pixels + cd.out_off + (size_t)x * 4,
             step, (int)cd.h, cd.blur_radius, i & 3, true);
}

// MaskFilterOnFilter's styles (mask_filter.cc:61-100) for the temp canvases
// that are not kNormal: the blurred image (out_off) against the unblurred
// one (px_off), per pixel, in place in out_off.  One thread per pixel; the
// grid's y is the temp canvas.
__global__ void k_blur_style(DevBatch b, const uint32_t* temps, uint32_t n_temp) {
  const uint32_t t = blockIdx.y;
  if (t >= n_temp) return;
  const CanvasDesc cd = b.canvases[temps[t]];
  if (cd.blur_style <= 1) return;
  const uint64_t n = (uint64_t)cd.w * cd.h;
  const uint32_t* raw = (const uint32_t*)(b.pixels + cd.px_off);
  uint32_t* out = (uint32_t*)(b.pixels + cd.out_off);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = ARGBtoRGBA(BlurStylePixel(cd.blur_style, RGBAtoARGB(raw[i]), RGBAtoARGB(out[i])));
}

__global__ void __launch_bounds__(kBlurThreads)
    k_blur_h_staged(DevBatch b, const uint32_t* temps, uint32_t n_temp) {
  extern __shared__ uint32_t bsm[];
  const uint32_t t = blockIdx.y;
  if (t >= n_temp) return;
  const CanvasDesc cd = b.canvases[temps[t]];
  const uint32_t rows = BlurRowsPerBlock(cd.w);
  if (rows == 0 || cd.blur_style == 0) return;  // direct pass, or a layer (no blur)
  const uint32_t y0 = blockIdx.x * rows;
  if (y0 >= cd.h) return;
  const uint32_t nr = min(rows, cd.h - y0);
  const uint32_t ws = OddStride(cd.w);
  uint32_t* in = bsm;
  uint32_t* out = bsm + rows * ws;
  const uint32_t* src = (const uint32_t*)(b.pixels + cd.px_off) + (size_t)y0 * cd.w;
  uint32_t* dst = (uint32_t*)(b.pixels + cd.blur_off) + (size_t)y0 * cd.w;
  const uint32_t n = nr * cd.w;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) in[(i / cd.w) * ws + i % cd.w] = src[i];
  __syncthreads();
  const uint32_t line = threadIdx.x >> 2;
  if (line < nr)
    BlurOrCopy((const uint8_t*)(in + line * ws), 4, (uint8_t*)(out + line * ws), 4, (int)cd.w,
               cd.blur_radius, threadIdx.x & 3, false);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = out[(i / cd.w) * ws + i % cd.w];
}

__global__ void __launch_bounds__(kBlurStripThreads)
    k_blur_v_staged(DevBatch b, const uint32_t* temps, uint32_t n_temp) {
  extern __shared__ uint32_t bsm[];
  const uint32_t t = blockIdx.y;
  if (t >= n_temp) return;
  const CanvasDesc cd = b.canvases[temps[t]];
  if (!BlurStripFits(cd.h) || cd.blur_style == 0) return;  // direct pass, or a layer
  const uint32_t x0 = blockIdx.x * kBlurStrip;
  if (x0 >= cd.w) return;
  const uint32_t nc = min((uint32_t)kBlurStrip, cd.w - x0);
  const uint32_t ws = OddStride(kBlurStrip);
  const uint32_t* src = (const uint32_t*)(b.pixels + cd.blur_off) + x0;
  const uint32_t lane = threadIdx.x % kBlurStrip;
  for (uint32_t y = threadIdx.x / kBlurStrip; y < cd.h; y += 4)
    if (lane < nc) bsm[y * ws + lane] = src[(size_t)y * cd.w + lane];
  __syncthreads();
  const uint32_t col = threadIdx.x >> 2;
  if (col >= nc) return;
  BlurOrCopy((const uint8_t*)(bsm + col), 4 * ws, b.pixels + cd.out_off + 4 * (size_t)(x0 + col),
             4 * (size_t)cd.w, (int)cd.h, cd.blur_radius, threadIdx.x & 3, true);
}

int LaunchBlur(const DevBatch& b, const uint32_t* temps, uint32_t n_temp, uint32_t max_h,
               uint32_t max_w, uint32_t max_style, cudaStream_t stream) {
  // no blurred temp canvases (the temps are layers): nothing to blur
  if (n_temp == 0 || max_w == 0 || max_h == 0) return 0;
  // staged passes (their blocks for canvases that do not fit return at once)
  const uint32_t min_rows = std::max<uint32_t>(BlurRowsPerBlock(max_w), 1);
  dim3 gsh((max_h + min_rows - 1) / min_rows, n_temp);
  const uint32_t smem_h = std::min<uint32_t>(2u * kBlurRows * OddStride(max_w), kBlurSmemWords);
  k_blur_h_staged<<<gsh, kBlurThreads, smem_h * 4, stream>>>(b, temps, n_temp);
  // direct passes for the canvases the staged ones do not take
  int n = 1;
  if (BlurRowsPerBlock(max_w) == 0) {
    dim3 gh((max_h + 31) / 32, n_temp);
    k_blur_h<<<gh, 128, 0, stream>>>(b, temps, n_temp);
    n++;
  }
  dim3 gsv((max_w + kBlurStrip - 1) / kBlurStrip, n_temp);
  const uint32_t smem_v =
      (uint32_t)std::min<uint64_t>((uint64_t)OddStride(kBlurStrip) * max_h, kBlurSmemWords);
  k_blur_v_staged<<<gsv, kBlurStripThreads, smem_v * 4, stream>>>(b, temps, n_temp);
  n++;
  if (!BlurStripFits(max_h)) {
    dim3 gv((max_w + 31) / 32, n_temp);
    k_blur_v<<<gv, 128, 0, stream>>>(b, temps, n_temp);
    n++;
  }
  if (max_style <= 1) return n;  // kNormal blurs in place: nothing to combine
  const uint64_t px = (uint64_t)max_w * max_h;
  dim3 gs((unsigned)std::min<uint64_t>((px + 255) / 256, 1024), n_temp);
  k_blur_style<<<gs, 256, 0, stream>>>(b, temps, n_temp);
  return n + 1;
}

}  // namespace skc

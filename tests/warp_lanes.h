// Test-only: the warp intrinsics the device code uses, on the CPU, so that it
// runs with 32 lanes here as it does on the GPU.  Each lane is a fiber; a
// collective waits until the 32 lanes of its warp have come to the same one,
// and lanes run in a random order between two collectives, so that a missing
// __syncwarp shows.  MeetWarps is the barrier of a pair of warps.  Include
// before the device headers.
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>
#include <vector_types.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

#undef __device__
#define __device__
#define __CUDA_ARCH__ 1030

namespace lanes32 {

constexpr size_t kStack = 512 << 10;
enum Op { kRun, kBallot, kSync, kShfl, kUp, kDown, kXor, kMin, kMax, kOr, kAdd, kMeet, kDone };
struct Fiber {
  ucontext_t at;
  std::vector<char> stack;
  Op op = kDone;
  unsigned gen = 0;
};
static Fiber fibers[64];
static uint64_t values[2][64];
static ucontext_t scheduler;
static int now = 0;  // the fiber that runs: 32 warp + lane
static const std::function<void(int, int)>* body;
static uint32_t order = 1;

static void Entry() {
  (*body)(now >> 5, now & 31);
  fibers[now].op = kDone;
  swapcontext(&fibers[now].at, &scheduler);
}
static void Wait(Op op) {
  fibers[now].op = op;
  swapcontext(&fibers[now].at, &scheduler);
}
// The lanes' values at this collective.
static inline const uint64_t* Collect(Op op, uint64_t v) {
  const int me = now;
  uint64_t* row = values[fibers[me].gen++ & 1];
  row[me] = v;
  Wait(op);
  return row + (me & 32);
}

// f(warp, lane) for the lanes of `warps` (1 or 2) warps.
static void Run(int warps, const std::function<void(int, int)>& f) {
  const int n = 32 * warps;
  body = &f;
  for (int i = 0; i < n; ++i) {
    Fiber& b = fibers[i];
    b.stack.resize(kStack);
    getcontext(&b.at);
    b.at.uc_stack.ss_sp = b.stack.data();
    b.at.uc_stack.ss_size = kStack;
    b.at.uc_link = nullptr;
    makecontext(&b.at, Entry, 0);
    b.op = kRun;
    b.gen = 0;
  }
  for (;;) {
    int lanes[64];
    for (int i = 0; i < n; ++i) lanes[i] = i;
    for (int i = n - 1; i > 0; --i) {
      order = order * 1664525u + 1013904223u;
      std::swap(lanes[i], lanes[(order >> 8) % (i + 1)]);
    }
    for (int j = 0; j < n; ++j) {
      now = lanes[j];
      if (fibers[now].op == kRun) swapcontext(&scheduler, &fibers[now].at);
    }
    bool done = true, meet = true;
    for (int w = 0; w < warps; ++w) {
      const Op op = fibers[32 * w].op;
      for (int i = 0; i < 32; ++i)
        if (fibers[32 * w + i].op != op) {
          std::fprintf(stderr, "warp %d: lane %d at op %d, lane 0 at %d\n", w, i,
                       fibers[32 * w + i].op, op);
          std::abort();
        }
      done = done && op == kDone;
      meet = meet && op == kMeet;
      if (op != kDone && op != kMeet)
        for (int i = 0; i < 32; ++i) fibers[32 * w + i].op = kRun;
    }
    if (done) return;
    if (meet)
      for (int i = 0; i < n; ++i) fibers[i].op = kRun;
    bool runs = false;
    for (int i = 0; i < n; ++i) runs = runs || fibers[i].op == kRun;
    if (!runs) {
      std::fprintf(stderr, "a warp waits for one that has ended\n");
      std::abort();
    }
  }
}
static inline void MeetWarps() { Wait(kMeet); }

template <typename T>
uint64_t Bits(T v) {
  uint64_t r = 0;
  std::memcpy(&r, &v, sizeof v);
  return r;
}
template <typename T>
T Value(uint64_t r) {
  T v;
  std::memcpy(&v, &r, sizeof v);
  return v;
}
template <typename T, typename F>
T Reduce(Op op, T v, F&& f) {
  const uint64_t* b = Collect(op, Bits(v));
  T r = Value<T>(b[0]);
  for (int i = 1; i < 32; ++i) r = f(r, Value<T>(b[i]));
  return r;
}

}  // namespace lanes32

static inline unsigned __ballot_sync(unsigned, bool p) {
  const uint64_t* b = lanes32::Collect(lanes32::kBallot, p);
  unsigned m = 0;
  for (int i = 0; i < 32; ++i) m |= (unsigned)(b[i] & 1) << i;
  return m;
}
static inline void __syncwarp(unsigned = 0) { lanes32::Collect(lanes32::kSync, 0); }
template <typename T>
T __shfl_sync(unsigned, T v, int src) {
  return lanes32::Value<T>(lanes32::Collect(lanes32::kShfl, lanes32::Bits(v))[src & 31]);
}
template <typename T>
T __shfl_up_sync(unsigned, T v, int o) {
  const int me = lanes32::now & 31;
  const uint64_t* b = lanes32::Collect(lanes32::kUp, lanes32::Bits(v));
  return me >= o ? lanes32::Value<T>(b[me - o]) : v;
}
template <typename T>
T __shfl_down_sync(unsigned, T v, int o) {
  const int me = lanes32::now & 31;
  const uint64_t* b = lanes32::Collect(lanes32::kDown, lanes32::Bits(v));
  return me + o < 32 ? lanes32::Value<T>(b[me + o]) : v;
}
template <typename T>
T __shfl_xor_sync(unsigned, T v, int o) {
  const int me = lanes32::now & 31;
  return lanes32::Value<T>(lanes32::Collect(lanes32::kXor, lanes32::Bits(v))[me ^ o]);
}
template <typename T>
T __reduce_min_sync(unsigned, T v) {
  return lanes32::Reduce(lanes32::kMin, v, [](T a, T b) { return std::min(a, b); });
}
template <typename T>
T __reduce_max_sync(unsigned, T v) {
  return lanes32::Reduce(lanes32::kMax, v, [](T a, T b) { return std::max(a, b); });
}
template <typename T>
T __reduce_or_sync(unsigned, T v) {
  return lanes32::Reduce(lanes32::kOr, v, [](T a, T b) { return a | b; });
}
template <typename T>
T __reduce_add_sync(unsigned, T v) {
  return lanes32::Reduce(lanes32::kAdd, v, [](T a, T b) { return a + b; });
}
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
static inline float rsqrtf(float v) { return 1.0f / std::sqrt(v); }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __saturatef(float v) { return v > 0 ? (v < 1 ? v : 1.f) : 0.f; }
static inline int __popc(unsigned v) { return __builtin_popcount(v); }
static inline int __ffs(int v) { return __builtin_ffs(v); }
static inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
template <typename T>
T atomicAdd(T* p, T v) {
  const T old = *p;
  *p += v;
  return old;
}
template <typename T>
T atomicOr(T* p, T v) {
  const T old = *p;
  *p |= v;
  return old;
}
using std::max;
using std::min;

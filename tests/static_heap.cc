// Test-only: how often skity_cuda_draw_path_static takes memory from the host
// heap, counted by this program's own operator new.  Arguments: path lengths;
// prints "length status allocations" for a draw of each, after a first draw.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "../include/skity_cuda.h"

static std::atomic<bool> armed{false};
static std::atomic<long> taken{0};

static void* Take(size_t n) {
  if (armed) ++taken;
  return std::malloc(n ? n : 1);
}
void* operator new(size_t n) {
  if (void* p = Take(n)) return p;
  throw std::bad_alloc();
}
void* operator new[](size_t n) { return operator new(n); }
void* operator new(size_t n, const std::nothrow_t&) noexcept { return Take(n); }
void* operator new[](size_t n, const std::nothrow_t&) noexcept { return Take(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }
void operator delete(void* p, const std::nothrow_t&) noexcept { std::free(p); }
void operator delete[](void* p, const std::nothrow_t&) noexcept { std::free(p); }

int main(int argc, char** argv) {
  uint8_t* canvas = nullptr;
  if (cudaMalloc((void**)&canvas, 256 * 256 * 4) != cudaSuccess) return 2;
  for (int a = 1; a < argc; ++a) {
    const uint32_t n = (uint32_t)std::atoi(argv[a]);
    std::vector<uint8_t> verbs(n, 1);
    std::vector<float> pts(2 * n);
    verbs[0] = 0;
    for (uint32_t i = 0; i < n; ++i) {
      pts[2 * i] = 128 + (40 + i % 60) * std::cos(6.2831853f * i / n);
      pts[2 * i + 1] = 128 + (40 + i % 60) * std::sin(6.2831853f * i / n);
    }
    skity_cuda_path path = {};
    path.verbs = verbs.data();
    path.verb_count = n;
    path.points = pts.data();
    path.point_count = n;
    skity_cuda_paint paint = {};
    paint.stroke_width = 1;
    paint.miter_limit = 4;
    paint.blend_mode = 3;
    paint.fill_color[0] = paint.fill_color[3] = 0.5f;
    int rc = skity_cuda_draw_path_static(0, canvas, 256, 256, 0, &path, &paint, nullptr);
    taken = 0;
    armed = true;
    if (!rc) rc = skity_cuda_draw_path_static(0, canvas, 256, 256, 0, &path, &paint, nullptr);
    armed = false;
    std::printf("%u %d %ld\n", n, rc, taken.load());
  }
  cudaFree(canvas);
  return 0;
}

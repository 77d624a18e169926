// Test-only: RunParts (batch.h) when the system gives no more memory while it
// starts its threads, and when a part throws.  Exits 0 when every part ran
// once whatever allocation failed, and when a part's exception came back after
// all threads had ended.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>

static thread_local long fail_at = -1;  // allocations of this thread until one fails

void* operator new(size_t n) {
  if (fail_at >= 0 && fail_at-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }

#include "../skity_gb300/csrc/batch.h"

int main() {
  constexpr uint32_t kParts = 500;
  for (unsigned threads : {1u, 2u, 9u, 32u}) {
    for (long k = -1; k < 80; ++k) {
      std::vector<std::atomic<int>> ran(kParts);
      fail_at = k;
      skc::RunParts(threads, kParts, [&](uint32_t r) { ++ran[r]; });
      fail_at = -1;
      for (auto& n : ran)
        if (n != 1) return 1;
    }
    std::atomic<int> done{0};
    bool thrown = false;
    try {
      skc::RunParts(threads, kParts, [&](uint32_t r) {
        if (r == 7) throw std::runtime_error("part 7");
        ++done;
      });
    } catch (const std::runtime_error&) {
      thrown = true;
    }
    const int at = done;
    if (!thrown || at < 7 || at != done) return 2;
  }
  std::puts("ok");
  return 0;
}

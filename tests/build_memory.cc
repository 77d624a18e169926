// Test-only: a stream build that runs out of host memory, at whichever
// allocation of whichever of its threads, gives the out-of-memory status.
// Arguments: threads, step, stream files.  Prints the allocations of a whole
// build and how many of the builds that were cut short gave the status;
// anything else exits 1.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

static std::atomic<long> left{-1};  // allocations until one fails (< 0: none does)
static std::atomic<long> made{0};

void* operator new(size_t n) {
  ++made;
  if (left >= 0 && left-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }

#include "../skity_gb300/csrc/batch.h"

int main(int argc, char** argv) {
  const unsigned threads = (unsigned)std::atoi(argv[1]);
  const long step = std::atol(argv[2]);
  std::vector<std::vector<uint8_t>> data;
  std::vector<const uint8_t*> streams;
  std::vector<size_t> bytes;
  for (int a = 3; a < argc; ++a) {
    std::FILE* f = std::fopen(argv[a], "rb");
    if (!f) return 1;
    std::vector<uint8_t> d;
    for (int c; (c = std::fgetc(f)) != EOF;) d.push_back((uint8_t)c);
    std::fclose(f);
    data.push_back(d);
  }
  for (auto& d : data) streams.push_back(d.data()), bytes.push_back(d.size());
  auto build = [&]() {
    skc::HostBatch hb;
    return skc::BuildStatus([&] {
      return skc::BuildStreams(hb, (uint32_t)data.size(), streams.data(), bytes.data(), threads);
    });
  };
  made = 0;
  if (build()) return 1;
  const long whole = made;
  long cut = 0;
  for (long k = 0; k < whole; k += step) {
    left = k;
    const int rc = build();
    left = -1;
    // a thread that is not started is no failure
    if (rc == SKITY_CUDA_ERROR_OUT_OF_HOST_MEMORY) ++cut;
    else if (rc) return 1;
  }
  std::printf("%ld %ld\n", whole, cut);
  return 0;
}

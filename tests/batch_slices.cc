// Test-only: the geometry slices of a batch (DeviceBatch::LayoutSlices and
// GrowSlices, device.h) over a fake of the few CUDA calls they make.  Exits 0
// when no two passes ever share a byte of scratch, else the number of the
// first check that fails.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../skity_gb300/csrc/device.h"

static bool copies_fail = false;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (copies_fail) return cudaErrorUnknown;
  std::memcpy(to, from, n);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
namespace skc {
int32_t CudaErr(cudaError_t e) { return e == cudaSuccess ? SKITY_CUDA_SUCCESS : SKITY_CUDA_ERROR_DEVICE; }
}  // namespace skc

using namespace skc;

// The slices are apart, inside the scratch, end by slices_end, and the device
// has them as they are.
static bool Apart(const DeviceBatch& db) {
  std::vector<std::pair<uint64_t, uint64_t>> at;
  for (const PassDesc& pd : db.hb.passes) {
    SliceLayout L;
    L.compute(pd.cap, sizeof(Edge));
    at.push_back({pd.slice_off, pd.slice_off + L.bytes});
  }
  std::sort(at.begin(), at.end());
  for (size_t i = 0; i + 1 < at.size(); ++i)
    if (at[i].second > at[i + 1].first) return false;
  return at.back().second <= db.slices_end && db.slices_end <= db.scratch.cap &&
         std::memcmp(db.passes.p, db.hb.passes.data(), at.size() * sizeof(PassDesc)) == 0;
}

int main() {
  std::mt19937 rng(5);
  DeviceBatch db;
  for (int round = 0; round < 20; ++round) {
    db.Reset();
    if (db.slices_end != 0 || !db.slices_dirty) return 1;
    for (int i = 0; i < 40; ++i) {
      PassDesc pd;
      std::memset(&pd, 0, sizeof pd);
      pd.flags = i % 2 ? kPassStroke : 0;
      for (int k = 0; k < 9; ++k) pd.cap[k] = (int32_t)(rng() % 400);
      DerivedCaps(pd.cap, i % 2);
      db.hb.passes.push_back(pd);
    }
    copies_fail = true;  // a renderer that fails before the passes are up
    if (!db.LayoutSlices(0, nullptr) || !db.slices_dirty) return 2;
    copies_fail = false;
    if (db.LayoutSlices(1, nullptr) != SKITY_CUDA_ERROR_OUT_OF_DEVICE_MEMORY) return 3;
    // one renderer lays the slices out and fails later; the next one finds
    // them standing and lets passes outgrow them, until there is no room
    if (db.LayoutSlices(0, nullptr) || !Apart(db)) return 4;
    bool again = false;
    for (int step = 0; step < 400 && !again; ++step) {
      if (db.LayoutSlices(0, nullptr)) return 5;
      db.h_geom.assign(40, PassGeom{});
      for (int i = 0; i < 3; ++i) {
        PassGeom& g = db.h_geom[rng() % 40];
        g.status = 1;
        g.need[rng() % 9] = (int32_t)(rng() % 2000);
      }
      std::vector<uint32_t> todo;
      if (db.GrowSlices(todo, nullptr)) return 6;
      size_t grown = 0;
      for (const PassGeom& g : db.h_geom) grown += g.status != 0;
      if (todo.size() != grown) return 7;
      again = db.slices_dirty;
      if (!again && !Apart(db)) return 8;
    }
    if (!again) return 9;
    if (db.LayoutSlices(0, nullptr) || !Apart(db)) return 10;
  }
  std::puts("ok");
  return 0;
}

// Test-only: the edge sort of a pass (edges.cuh) as the GPU runs it, by the 32
// lanes of a warp, and std::sort, which it has to follow among equal keys.
#include "warp_lanes.h"

#include "../skity_gb300/csrc/edges.cuh"

using namespace skc;

// The sort of EdgesPass: keys on chip up to kSortKeys edges, else in scratch.
extern "C" void skc_lanes_sort(const int32_t* y, const int32_t* x, const int32_t* dx, int32_t* idx,
                               int n) {
  static SortShared sh;
  std::vector<SortKey> scratch(n);
  SortKey* keys = n <= kSortKeys ? sh.keys : scratch.data();
  lanes32::Run(1, [&](int, int lane) {
    Lanes L;
    L.lane = lane;
    for (int i = lane; i < n; i += 32) {
      keys[i].y = y[i];
      keys[i].x = x[i];
      keys[i].dx = dx[i];
      keys[i].idx = i;
    }
    L.sync();
    SortKeyLess less;
    IntrosortPartitions(L, &sh, keys, n, less);
    for (int i = lane; i < n; i += 32) idx[StableRank(keys, n, i, less)] = keys[i].idx;
  });
}

extern "C" void skc_std_sort_edges(const int32_t* y, const int32_t* x, const int32_t* dx,
                                   int32_t* idx, int n) {
  std::vector<SortKey> keys(n);
  for (int i = 0; i < n; ++i) keys[i] = {y[i], x[i], dx[i], i};
  std::sort(keys.begin(), keys.end(), [](const SortKey& a, const SortKey& b) {
    return a.y != b.y ? a.y < b.y : a.x != b.x ? a.x < b.x : a.dx < b.dx;
  });
  for (int i = 0; i < n; ++i) idx[i] = keys[i].idx;
}

// Keys on which std::sort partitions badly, until it falls back to its heap
// sort: values are settled only as the sort compares them (M. D. McIlroy, "A
// Killer Adversary for Quicksort", 1999).
extern "C" void skc_adversary(int32_t* keys, int n) {
  std::vector<int> v(n), at(n);
  int solid = 0, candidate = 0;
  const int gas = n;
  for (int i = 0; i < n; ++i) v[i] = gas, at[i] = i;
  std::sort(at.begin(), at.end(), [&](int a, int b) {
    if (v[a] == gas && v[b] == gas) {
      if (a == candidate) v[a] = solid++;
      else v[b] = solid++;
    }
    if (v[a] == gas) candidate = a;
    else if (v[b] == gas) candidate = b;
    return v[a] < v[b];
  });
  for (int i = 0; i < n; ++i) keys[i] = v[i];
}

// MaxActive over edges sorted by upper_y, and the same bound by counting.
extern "C" void skc_max_active(const int32_t* upper, const int32_t* lower, int n, int32_t out[2]) {
  static SortShared sh;
  std::vector<Edge> edges(n);
  std::vector<int32_t> tmp(2 * n + 2);
  for (int i = 0; i < n; ++i) {
    std::memset(&edges[i], 0, sizeof(Edge));
    edges[i].upper_y = upper[i];
    edges[i].lower_y = lower[i];
  }
  lanes32::Run(1, [&](int, int lane) {
    Lanes L;
    L.lane = lane;
    const int got = MaxActive(L, &sh, edges.data(), n, tmp.data());
    if (lane == 0) out[0] = got;
  });
  out[1] = 0;
  for (int i = 0; i < n; ++i) {
    int c = 0;
    for (int j = 0; j <= i; ++j) c += lower[j] > upper[i];
    out[1] = std::max(out[1], c);
  }
}

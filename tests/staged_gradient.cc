// Test-only: the compositor's staged gradient colour (composite.cuh,
// GradientColorStaged) against the general one (GradientColor) on the CPU.
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

#include "../skity_gb300/csrc/kernels.cuh"

using namespace skc;

// Random gradients of 2 to 16 stops the staged form takes, every tile mode, at
// parameters on, beside and between the stops and the cells; returns the
// number of differing colours, and the number compared in *compared.
extern "C" int64_t staged_gradient_check(uint32_t seed, int gradients, int64_t* compared) {
  std::mt19937 rng(seed);
  auto uni = [&](float lo, float hi) { return std::uniform_real_distribution<float>(lo, hi)(rng); };
  int64_t bad = 0;
  *compared = 0;
  for (int g = 0; g < gradients; ++g) {
    const int n = 2 + (int)(rng() % 15);
    const int form = (int)(rng() % 5);
    std::vector<float4> col(n);
    std::vector<float> off(n), recip(n + 1);
    for (auto& c : col) {
      const float lo = form == 4 ? -0.5f : 0.f, hi = form == 4 ? 1.5f : 1.f;
      c.x = uni(lo, hi), c.y = uni(lo, hi), c.z = uni(lo, hi), c.w = uni(lo, hi);
      if (rng() % 4 == 0) c.w = 1.f;
    }
    float last = form == 3 ? -1.5f : 0.f;
    for (int i = 0; i < n; ++i) {
      if (form == 0) off[i] = i ? uni(0, 1) : 0.f;
      else if (form == 1) off[i] = (float)(rng() % 33) / 32;  // on cell borders, some equal
      else if (form == 2) off[i] = last += (rng() % 3 ? 1e-6f : 0.4f) * uni(0.96f, 1.f);
      else off[i] = last += uni(0.f, 0.4f);
    }
    for (int i = 1; i < n; ++i)
      for (int j = i; j > 0 && off[j] < off[j - 1]; --j) std::swap(off[j], off[j - 1]);
    bool fits = true;
    for (int i = 0; i < n; ++i) fits = fits && StagedStop(col[i], off[i], i + 1 < n ? off[i + 1] : off[i]);
    if (!fits) continue;
    for (int i = 0; i < n; ++i) recip[i] = 1.0f / ((i + 1 < n ? off[i + 1] : off[i]) - off[i]);
    uint8_t first[32];
    for (int c = 0; c < 32; ++c) first[c] = (uint8_t)FirstInterval(off.data(), n, c);
    StagedStops st{col.data(), off.data(), recip.data(), first};
    Brush b{};
    b.stop_count = (uint32_t)n;
    b.has_offsets = 1;
    std::vector<float> at{-2.f, -1.f, -0.f, 0.f, 1e-30f, 0.5f, 1.f, 1.0000001f, 2.f, 3.5f};
    for (float o : off)
      for (float v : {o, std::nextafterf(o, -9.f), std::nextafterf(o, 9.f), o + 1e-20f}) at.push_back(v);
    for (int c = 0; c <= 32; ++c)
      for (float v : {c / 32.f, std::nextafterf(c / 32.f, -9.f), std::nextafterf(c / 32.f, 9.f)}) at.push_back(v);
    for (int k = 0; k < 200; ++k) at.push_back(uni(-1.5f, 2.5f));
    for (uint32_t tile = 0; tile < 4; ++tile) {
      b.tile = tile;
      for (float t : at) {
        ++*compared;
        if (GradientColor(b, t, col.data(), off.data()) != GradientColorStaged(tile, n, t, st)) ++bad;
      }
    }
  }
  return bad;
}

// value / total by the reciprocal against the division.
extern "C" int64_t div_by_recip_check(uint32_t seed, int64_t count) {
  std::mt19937 rng(seed);
  int64_t bad = 0;
  for (int64_t i = 0; i < count; ++i) {
    const float total = std::ldexp(1.f + (rng() >> 8) * 0x1p-24f, -20 + (int)(rng() % 23));
    float value = rng() % 2 ? total * ((rng() >> 8) * 0x1p-24f)
                            : std::ldexp(1.f + (rng() >> 8) * 0x1p-24f, -49 + (int)(rng() % 52));
    if (!(value <= total) || value < 1e-15f) continue;
    if (DivByRecip(value, total, 1.0f / total) != value / total) ++bad;
  }
  return bad;
}

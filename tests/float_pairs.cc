// Test-only: the float-pair arithmetic of the stroker and the curve counts
// against the double arithmetic it stands for, on the CPU.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#include "../skity_gb300/csrc/kernels.cuh"
#include "../skity_gb300/csrc/stroke.cuh"

using namespace skc;

static bool Same(float a, float b) { return std::memcmp(&a, &b, 4) == 0 || (std::isnan(a) && std::isnan(b)); }

// counts[0..3]: differing results of PointSetLength, FindUnitQuadRoots'
// discriminant, CubicQuadCountD and the mirror tile; counts[4..5]: how often
// the pairs settled the first two.
extern "C" void float_pairs_check(uint32_t seed, int64_t n, int64_t counts[6]) {
  std::mt19937 rng(seed);
  auto val = [&](int form) {
    const float m = 1.f + (rng() >> 8) * 0x1p-24f;
    const float s = rng() & 1 ? 1.f : -1.f;
    if (form == 0) return s * std::ldexp(m, (int)(rng() % 24) - 10);
    if (form == 1) return s * std::ldexp(m, (int)(rng() % 120) - 60);
    if (form == 2) return s * (float)(rng() % 2000) * 0.25f;
    return rng() % 3 ? s * m : 0.f * s;
  };
  for (int k = 0; k < 6; ++k) counts[k] = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int form = (int)(rng() % 4);
    const float x = val(form), y = val(form), len = i % 3 ? std::fabs(val(2)) + 0.125f : 1.0f;
    P a, b;
    const bool ra = PointSetLength(&a, x, y, len), rb = PointSetLengthDouble(&b, x, y, len);
    if (ra != rb || !Same(a.x, b.x) || !Same(a.y, b.y)) counts[0]++;
    const float A = val(form), B = val(form), C = val(form);
    float r;
    if (DiscriminantRoot(A, B, C, &r)) {
      counts[5]++;
      if (!Same(r, (float)std::sqrt((double)B * B - 4 * (double)A * C))) counts[1]++;
    }
    P c[4];
    for (auto& q : c) q = mkP(val(form == 1 ? 0 : form), val(form == 1 ? 0 : form));
    {
      const float acc = 0.1f;
      const double mh = 432.0 * acc * acc;
      const P p = mkP(c[1].x * 3.f - c[0].x, c[1].y * 3.f - c[0].y);
      const P q = mkP(c[2].x * 3.f - c[3].x, c[2].y * 3.f - c[3].y);
      const P d = mkP(q.x - p.x, q.y - p.y);
      const float err = d.x * d.x + d.y * d.y;
      const double want = std::max(1., std::ceil(std::pow(err / mh, 1. / 6.0)));
      if (CubicQuadCountD(c) != want) counts[2]++;
    }
    const float t = val(form), t1 = t - 1;
    const float want = std::fabs((float)((double)t1 - 2.0 * std::floor((double)t1 * 0.5) - 1.0));
    if (!Same(RemapFloatTile(t, 2), want)) counts[3]++;
  }
}

// (float)(i / n) in double against the float division, every i <= n < limit.
extern "C" int64_t quad_ends_check(int limit) {
  int64_t bad = 0;
  for (int n = 1; n < limit; ++n)
    for (int i = 0; i <= n; ++i)
      if ((float)((double)i / n) != (float)i / (float)n) ++bad;
  return bad;
}

// The triangle test's double-precision redo in its two forms (ubr_internal.h)
// against the plain sum, bit for bit: random triangles, and rays through
// vertices and edges, where an edge function is zero.
#include <cstdio>
#include <cstring>
#include <random>

#include "ubr_internal.h"

using namespace ubr;

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok && ++failures < 20) std::printf("FAILED: %s\n", what);
}
static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0; }

int main() {
  std::mt19937 rng(5);
  auto u = [&] { return float(int(rng() % 2001) - 1000) * 0.001f; };
  int zero = 0, hits = 0;
  for (int k = 0; k < 400000; ++k) {
    // integer and half coordinates now and then, so products cancel exactly
    const bool grid = k % 2 == 0;
    auto c = [&] { return grid ? 0.5f * float(int(rng() % 9) - 4) : u(); };
    f3 v[3];
    for (f3& p : v) p = f3{c(), c(), c()};
    f3 target = v[rng() % 3];
    if (k % 3 == 0) target = (v[0] + v[1]) * 0.5f;
    if (k % 3 == 1) target = f3{c(), c(), c()};
    const f3 org{c(), c(), c() + 6.0f};
    const f3 dir = k % 5 == 0 ? f3{0.0f, 0.0f, -1.0f} : target - org;
    const TriPre pre = triPre(dir, org);
    const float X[3][3] = {{v[0].x, v[1].x, v[2].x}, {v[0].y, v[1].y, v[2].y}, {v[0].z, v[1].z, v[2].z}};
    auto row = [&](int a) { return make_float4(X[a][0], X[a][1], X[a][2], 0.0f); };
    const float4 rx = row(pre.kx), ry = row(pre.ky), rz = row(pre.kz);
    Hit a{}, b{};
    const bool ha = isectTriangle<false>(pre, rx, ry, rz, 0.0f, 1e30f, a);
    const bool hb = isectTriangle<true>(pre, rx, ry, rz, 0.0f, 1e30f, b);
    check(ha == hb, "the same answer");
    hits += ha;
    if (!ha) continue;
    check(same(a.t, b.t) && same(a.u, b.u) && same(a.v, b.v), "the same hit");
    zero += a.u == 0.0f || a.v == 0.0f || a.u + a.v == 1.0f;
  }
  check(hits > 10000 && zero > 1000, "hits, many of them on an edge");
  if (failures) std::printf("%d failures\n", failures);
  return failures ? 1 : 0;
}

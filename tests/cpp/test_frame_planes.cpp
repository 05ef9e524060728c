// The choice of the planes a call writes in place (csrc/frame_planes.h) against
// a check of every pair.
#include <cstdio>
#include <random>

#include "frame_planes.h"

using ubr::PlaneUse;

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok && ++failures < 20) std::printf("FAILED: %s\n", what);
}
static const void* at(uintptr_t a) { return reinterpret_cast<const void*>(a); }

int main() {
  std::mt19937 rng(7);
  for (int round = 0; round < 20000; ++round) {
    const int n = int(rng() % 14);
    const uintptr_t span = 16u << (rng() % 12);  // dense to sparse
    std::vector<PlaneUse> in;
    for (int k = 0; k < n; ++k) {
      const bool none = rng() % 6 == 0;
      const size_t align = rng() % 5 == 0 ? 0 : rng() % 4 == 0 ? 16 : 4;
      const uintptr_t odd = rng() % 8 == 0 ? 1 + rng() % 15 : 0;
      in.push_back(PlaneUse{none ? nullptr : at(4096 + 4 * (rng() % span) + odd), 4 * size_t(rng() % 40), align,
                            rng() % 2 == 0});
    }
    std::vector<PlaneUse> out = in;
    // memory of the device ends at `top`; a plane that is null, empty or not
    // aligned needs no look at it
    const uintptr_t top = 4096 + 4 * (rng() % (span + 40));
    auto ours = [&](const void* q, size_t bytes) {
      check(q && bytes, "asked for a plane that is not there");
      return reinterpret_cast<uintptr_t>(q) + bytes <= top;
    };
    choosePlanes(out, ours);
    for (int i = 0; i < n; ++i) {
      const uintptr_t a = reinterpret_cast<uintptr_t>(in[i].ptr);
      bool want = in[i].align && in[i].ptr && in[i].bytes && a % in[i].align == 0 && a + in[i].bytes <= top;
      for (int j = 0; j < n; ++j) {
        const uintptr_t c = reinterpret_cast<uintptr_t>(in[j].ptr);
        if (i != j && in[i].ptr && in[j].ptr && in[i].bytes && in[j].bytes && a < c + in[j].bytes &&
            c < a + in[i].bytes)
          want = false;
      }
      check(out[i].inPlace == want, "aligned planes on the device that meet no other, and only they, are written in place");
      check(out[i].ptr == in[i].ptr && out[i].bytes == in[i].bytes, "order and extents are kept");
    }
  }
  // known ranges answer as the driver would, asked once per allocation: blocks
  // of 64 to 191 bytes every 192 bytes from 4096 on, some of other memory
  for (int round = 0; round < 2000; ++round) {
    ubr::KnownRanges known;
    const unsigned salt = rng();
    int asked = 0;
    std::vector<int> met(64, 0);
    for (int k = 0; k < 60; ++k) {
      const uintptr_t a = 4096 + rng() % (192 * 64);
      const size_t bytes = rng() % 200, block = (a - 4096) / 192;
      const uintptr_t start = 4096 + 192 * block;
      const size_t size = 64 + (salt * (unsigned(block) + 7u) >> 5) % 128;
      const bool ours = (salt >> (block % 32)) & 1u;
      auto ask = [&](uintptr_t& s, size_t& n) {
        ++asked;
        check(++met[block] == 1 || !ours || a >= start + size, "asked once for an allocation");
        s = start;
        n = size;
        return ours && a < start + size;
      };
      if (ours && a >= start + size) met[block] -= 1;  // between the allocations: asked again
      const bool got = known(at(a), bytes, ask);
      check(got == (ours && a < start + size && a + bytes <= start + size), "within one allocation of ours");
    }
    check(asked > 0, "the driver was asked");
  }
  if (failures) std::printf("%d failures\n", failures);
  return failures ? 1 : 0;
}

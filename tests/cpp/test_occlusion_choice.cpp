// Which launches of occlusion rays run the kernel whose warps fetch rays
// (csrc/occlusion_choice.h).
#include <cstdio>
#include <initializer_list>

#include "occlusion_choice.h"

using ubr::chooseFetch;

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok && ++failures < 20) std::printf("FAILED: %s\n", what);
}

int main() {
  // around the line, in one or many rays per hit
  for (const uint64_t R : {1, 3, 13, 17, 64}) {
    const uint64_t n = (ubr::kFetchRays + R - 1) / R;
    check(chooseFetch(0, false, false, n, R), "at the line");
    check(!chooseFetch(0, false, false, n - 1, R), "below the line");
    check(!chooseFetch(0, true, false, n, R), "triangles");
    check(!chooseFetch(0, false, true, n, R), "nearest hits");
  }
  check(chooseFetch(0, false, false, 3000000000u, 3000), "more rays than 32 bits count");
  check(!chooseFetch(0, false, false, 0, 64) && !chooseFetch(0, false, false, 1000, 0), "no rays");
  // the launches whose pictures are compared with one thread per ray: {pixels,
  // rays per hit, fetched}
  const struct { uint64_t n, R; bool fetch; } launches[] = {
      {1000 * 705, 16 + 1, false}, {1001 * 707, 16 + 1, true}, {1283 * 721, 13, true},
      {999 * 667, 16 + 2, false},  {1001 * 667, 16 + 2, true}, {641 * 479 * 4, 37 + 2, true}, {1400 * 1000, 7 + 2, true},
      {700 * 613 + 811 * 600 + 257 * 255 + 640 * 480, 16 + 2, true}, {901 * 853, 16 + 2, true}};
  for (const auto& l : launches) check(chooseFetch(0, false, false, l.n, l.R) == l.fetch, "a compared launch");
  // a context's own choice stands at any size
  for (int mode = 1; mode <= 4; ++mode)
    for (uint64_t n : {uint64_t(1), uint64_t(100000000)})
      for (int k = 0; k < 4; ++k)
        check(chooseFetch(mode, k & 1, k & 2, n, 18) == (mode == 2), "the context's choice");
  return failures ? 1 : 0;
}

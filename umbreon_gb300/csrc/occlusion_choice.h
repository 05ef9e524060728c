// occlusion_choice.h -- which kernel a launch of occlusion rays runs (host code
// only).
#pragma once

#include <cstdint>

namespace ubr {

// Whether a launch of n hits' rays (R each, n counting the misses too, as the
// host knows it) runs the persistent kernel: binary answers, spheres and
// cylinders only (with triangles the larger ray state costs 5-10 %), and
// enough rays.  Ball-and-stick of 5 k atoms, one thread per ray against the
// persistent kernel: 640x480 with 18 rays (5.5 M) 0.353 / 0.378 ms, 800x600
// (8.6 M) 0.501 / 0.510, 1024x768 (14 M) 0.723 / 0.700, 1280x720 ss2 (66 M)
// 2.61 / 2.26.
// mode: the context's trace_mode; mesh: the launch's kinds include triangles;
// nearest: some frame wants its AO rays' nearest hits.
constexpr uint64_t kFetchRays = 12000000;
inline bool chooseFetch(int mode, bool mesh, bool nearest, uint64_t n, uint64_t R) {
  if (mode != 0) return mode == 2;
  return !nearest && !mesh && n * R >= kFetchRays;
}

}  // namespace ubr

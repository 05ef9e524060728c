// frame_planes.h -- which of the caller's device planes a call writes as it
// renders (host code only).
//
// A plane written in place is also read back: later transparency layers ask
// the depth plane whether a pixel had its first hit, the fog reads view z, the
// denoiser reads the colour and the AOVs.  That is only right for memory that
// belongs to one plane of one frame.  The other planes are shaded into the
// context's buffers and copied at the end of the call, in the order of the
// frames, so planes that share memory end up as the last copy leaves them.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ubr {

struct PlaneUse {
  const void* ptr;  // null: not asked for
  size_t bytes;
  size_t align;     // of the kernels' stores; 0: the call only copies this plane
  bool inPlace;     // out: the call may write it as it renders
};

// A plane is written in place unless its memory meets another plane's, or it
// starts between two of the kernels' elements (a copy takes any address, a
// kernel's store there is a fault), or ours(ptr, bytes) does not know it as
// memory of the device in its whole length (a copy to other memory works, or
// fails with an error; a kernel's store would be a fault).
template <class Ours>
void choosePlanes(std::vector<PlaneUse>& planes, Ours&& ours) {
  std::vector<PlaneUse*> by;
  by.reserve(planes.size());
  auto at = [](const PlaneUse* u) { return reinterpret_cast<uintptr_t>(u->ptr); };
  for (PlaneUse& u : planes) {
    const bool some = u.ptr && u.bytes;
    u.inPlace = some && u.align && at(&u) % u.align == 0 && ours(u.ptr, u.bytes);
    if (some) by.push_back(&u);
  }
  std::sort(by.begin(), by.end(), [&](const PlaneUse* a, const PlaneUse* b) { return at(a) < at(b); });
  uintptr_t end = 0;  // of the planes so far
  for (size_t k = 0; k < by.size(); ++k) {
    if (at(by[k]) < end) by[k]->inPlace = by[k - 1]->inPlace = false;
    end = std::max(end, at(by[k]) + by[k]->bytes);
  }
}

// Allocations that a call has met, so that planes of one allocation cost one
// question to the driver (70 ns: 8 us of a batch of 24 frames with 120 planes).
// Not kept between calls.
class KnownRanges {
 public:
  // Whether [ptr, ptr + bytes) lies within one allocation; ask(start, size)
  // finds the one at ptr, or is false.
  template <class Ask>
  bool operator()(const void* ptr, size_t bytes, Ask&& ask) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(ptr);
    for (const Range& r : ranges_)
      if (r.holds(at)) return r.holds(at, bytes);
    Range r{};
    if (!ask(r.start, r.size) || !r.holds(at)) return false;
    ranges_.push_back(r);
    return r.holds(at, bytes);
  }

 private:
  struct Range {
    uintptr_t start;
    size_t size;
    bool holds(uintptr_t at, size_t bytes = 0) const {
      return at >= start && at - start < size && bytes <= size - (at - start);
    }
  };
  std::vector<Range> ranges_;
};

}  // namespace ubr

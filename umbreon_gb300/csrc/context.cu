// context.cu -- the context's errors and its device memory: allocations under
// the arena cap, the scratch that calls share, and workspaces (host code).
#include <algorithm>
#include <string>
#include <vector>

#include "ubr_context.h"

namespace ubr {

ubr_status setError(Context* c, ubr_status s, const std::string& msg) {
  if (c) c->lastError = msg;
  return s;
}

ubr_status cudaFail(Context* c, cudaError_t e, const char* what) {
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  cudaGetLastError();  // clear a non-sticky error so the context stays usable
  return setError(c, e == cudaErrorMemoryAllocation ? UBR_OUT_OF_MEMORY : UBR_CUDA_ERROR, m);
}

bool arenaHolds(const Context* c, size_t bytes) {
  return !c->arenaCap || bytes <= c->arenaCap - c->arenaUsed;
}

// Makes room for `bytes` under the arena cap: scratch that the running call has
// not asked for goes, workspaces first, then the largest.  Frees are ordered
// after the work in flight, and a captured graph's key holds the scratch that
// its launches use, so it is captured again when they have moved.
static void releaseIdle(Context* c, size_t bytes) {
  while (!arenaHolds(c, bytes)) {
    int pick = -1;
    auto rank = [&](int i) {
      const bool workspace = i == kGatherSlot || i == kAdjointSlot;
      return std::make_pair(workspace, c->scratch[size_t(i)].bytes);
    };
    for (int i = 0; i < int(c->scratch.size()); ++i) {
      const DevBuf& b = c->scratch[size_t(i)];
      if (b.ptr && b.call != c->call && (pick < 0 || rank(i) > rank(pick))) pick = i;
    }
    if (pick < 0) return;
    devFree(c, c->scratch[size_t(pick)]);
  }
}

ubr_status devAlloc(Context* c, DevBuf& b, size_t bytes, bool direct) {
  if (bytes == 0) bytes = 16;
  if (!arenaHolds(c, bytes)) releaseIdle(c, bytes);
  if (!arenaHolds(c, bytes)) return setError(c, UBR_OUT_OF_MEMORY, "device arena cap exceeded");
  void* p = nullptr;
  // stream-ordered from the context's pool: after the first frames a scene
  // build or a scratch growth reuses pooled memory instead of cudaMalloc
  b.direct = direct || !c->pool;
  cudaError_t e = b.direct ? cudaMalloc(&p, bytes) : cudaMallocFromPoolAsync(&p, bytes, c->pool, c->stream);
  if (e != cudaSuccess) return cudaFail(c, e, "device allocation");
  b.ptr = p;
  b.bytes = bytes;
  c->arenaUsed += bytes;
  return UBR_OK;
}

// A block of the slab, or null where none fits (first fit).
static void* slabCut(Slab& s, size_t bytes) {
  for (auto it = s.free.begin(); it != s.free.end(); ++it) {
    if (it->second < bytes) continue;
    void* p = static_cast<char*>(s.ptr) + it->first;
    it->first += bytes;
    it->second -= bytes;
    if (it->second == 0) s.free.erase(it);
    return p;
  }
  return nullptr;
}

static void slabDrop(Slab& s) {
  cudaFree(s.ptr);
  s = Slab{};
}

static void slabGive(Slab& s, void* p, size_t bytes) {
  const size_t at = size_t(static_cast<char*>(p) - static_cast<char*>(s.ptr));
  auto it = std::lower_bound(s.free.begin(), s.free.end(), std::make_pair(at, size_t(0)));
  it = s.free.insert(it, {at, bytes});
  if (it + 1 != s.free.end() && it->first + it->second == (it + 1)->first) {
    it->second += (it + 1)->second;
    s.free.erase(it + 1);
  }
  if (it != s.free.begin() && (it - 1)->first + (it - 1)->second == it->first) {
    (it - 1)->second += it->second;
    s.free.erase(it);
  }
  if (s.free[0].second == s.bytes) slabDrop(s);
}

void devFree(Context* c, DevBuf& b) {
  if (b.ptr) {
    if (b.slab) slabGive(c->slab, b.ptr, b.bytes);
    else if (b.direct) cudaFree(b.ptr);
    else cudaFreeAsync(b.ptr, c->stream);
    c->arenaUsed -= b.bytes;
  }
  b.ptr = nullptr;
  b.bytes = 0;
  b.slab = false;
}

// Scratch blocks from this size on come from cudaMalloc: a new pool grows by
// about 65 us plus 0.8 us per MB (128 MB 155 us, 512 MB 460 us), cudaMalloc
// takes 60-110 us at any size, and a block of the scratch lives as long as its
// context.  Scenes stay in the pool, which hands freed blocks on in 2 us.
constexpr size_t kDirectBytes = size_t(96) << 20;

static size_t withSlack(size_t bytes) { return bytes + bytes / 4; }
static size_t slabPadded(size_t bytes) { return (bytes + 255) / 256 * 256; }

ubr_status scratchGet(Context* c, int i, size_t bytes, void** out, bool slack) {
  if (size_t(i) >= c->scratch.size()) c->scratch.resize(size_t(i) + 1);
  DevBuf& b = c->scratch[size_t(i)];
  if (b.bytes < bytes) {
    // grow geometrically; wait for in-flight users of the old block first
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cudaFail(c, e, "cudaStreamSynchronize");
    devFree(c, b);
    const size_t grown = slack ? withSlack(bytes) : bytes;
    // small blocks stay out of the slab: many never grow, and one of them would
    // hold all of it
    void* cut = grown >= kSlabBlock ? slabCut(c->slab, slabPadded(grown)) : nullptr;
    if (cut) {
      b.ptr = cut;
      b.bytes = slabPadded(grown);
      b.slab = true;
      c->arenaUsed += b.bytes;
    } else {
      ubr_status st = devAlloc(c, b, grown, grown >= kDirectBytes);
      // what the cap has no room for with the slack it may have without
      if (st == UBR_OUT_OF_MEMORY && c->arenaCap && bytes < grown) st = devAlloc(c, b, bytes, bytes >= kDirectBytes);
      if (st != UBR_OK) return st;
    }
  }
  b.call = c->call;
  *out = b.ptr;
  return UBR_OK;
}

// A context's first frame grows some thirty scratch blocks: 2-3 us each from
// the pool, 65 us whenever it has to grow (by 32 MB at least) and 0.8 us per MB;
// the slab is one cudaMalloc, worth it from about two growths on (first GI
// frames: 640x480 pt1 791 -> 726 us, 955x198 pt1 700 -> 598).
void scratchReserve(Context* c, const std::vector<ScratchNeed>& plan) {
  if (c->slab.ptr) {
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return;  // the next scratchGet reports it
    for (DevBuf& b : c->scratch)
      if (b.slab && b.call != c->call) devFree(c, b);
    if (c->slab.ptr && c->slab.free.size() == 1 && c->slab.free[0].second == c->slab.bytes) slabDrop(c->slab);
    if (c->slab.ptr) return;  // this call uses blocks of it already
  }
  size_t want = 0;
  for (const ScratchNeed& n : plan) {
    const size_t has = size_t(n.slot) < c->scratch.size() ? c->scratch[size_t(n.slot)].bytes : 0;
    const size_t grown = n.slack ? withSlack(n.bytes) : n.bytes;
    if (has < n.bytes && grown >= kSlabBlock) want += slabPadded(grown);
  }
  if (c->arenaCap != 0 || want < kSlabLeast || want > kSlabBytes) return;
  void* p = nullptr;
  if (cudaMalloc(&p, want) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  c->slab.ptr = p;
  c->slab.bytes = want;
  c->slab.free = {{0, want}};
}

void scratchDone(Context* c, int slot) {
  if (size_t(slot) < c->scratch.size()) c->scratch[size_t(slot)].call = 0;
}

ubr_status workspaceGet(Context* c, int slot, size_t least, void* lent, size_t lentBytes, void** out, size_t* bytes) {
  if (size_t(slot) >= c->scratch.size()) c->scratch.resize(size_t(slot) + 1);
  const size_t want = *bytes, own = c->scratch[size_t(slot)].bytes;
  // the largest block that the running call does not use
  for (size_t k = 0; k < c->scratch.size(); ++k) {
    const DevBuf& b = c->scratch[k];
    if (int(k) == slot || !b.ptr || b.call == c->call || b.bytes <= lentBytes) continue;
    lent = b.ptr;
    lentBytes = b.bytes;
  }
  // a block of its own: all it wants, or what the cap leaves where that is more
  // than there is without (by a quarter, lest it grow a little in every call)
  const size_t room = c->arenaCap ? c->arenaCap - c->arenaUsed + own : want, fit = std::min(want, room);
  if (own >= want || fit == want || (fit >= least && fit > lentBytes && fit > own + own / 4)) {
    *bytes = std::min(want, std::max(own, fit));
    if (scratchGet(c, slot, *bytes, out, false) == UBR_OK) return UBR_OK;
    cudaGetLastError();
  }
  if (c->scratch[size_t(slot)].bytes >= std::max(least, lentBytes)) {
    *bytes = c->scratch[size_t(slot)].bytes;
    return scratchGet(c, slot, *bytes, out, false);
  }
  if (lentBytes >= least) {
    *out = lent;
    *bytes = std::min(want, lentBytes);
    return UBR_OK;
  }
  *bytes = least;
  return scratchGet(c, slot, least, out, false);
}

}  // namespace ubr

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

ubr_status devAlloc(Context* c, DevBuf& b, size_t bytes, bool direct) {
  if (bytes == 0) bytes = 16;
  if (c->arenaCap && c->arenaUsed + bytes > c->arenaCap)
    return setError(c, UBR_OUT_OF_MEMORY, "device arena cap exceeded");
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

void devFree(Context* c, DevBuf& b) {
  if (b.ptr) {
    if (b.slab) {
      Slab& s = c->slabs[size_t(b.slab) - 1];
      if (--s.live == 0) {
        cudaFree(s.ptr);
        s = Slab{};
      }
    } else if (b.direct) {
      cudaFree(b.ptr);
    } else {
      cudaFreeAsync(b.ptr, c->stream);
    }
    c->arenaUsed -= b.bytes;
  }
  b.ptr = nullptr;
  b.bytes = 0;
  b.slab = 0;
}

// Scratch blocks from this size on come from cudaMalloc: a new pool grows by
// about 65 us plus 0.8 us per MB (128 MB 155 us, 512 MB 460 us), cudaMalloc
// takes 60-110 us at any size, and a block of the scratch lives as long as its
// context.  Scenes stay in the pool, which hands freed blocks on in 2 us.
constexpr size_t kDirectBytes = size_t(96) << 20;

ubr_status scratchGet(Context* c, int i, size_t bytes, void** out, bool slack) {
  if (size_t(i) >= c->scratch.size()) c->scratch.resize(size_t(i) + 1);
  DevBuf& b = c->scratch[size_t(i)];
  if (b.bytes < bytes) {
    // grow geometrically; wait for in-flight users of the old block first
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cudaFail(c, e, "cudaStreamSynchronize");
    devFree(c, b);
    const size_t grown = slack ? bytes + bytes / 4 : bytes;
    const size_t padded = (grown + 255) / 256 * 256;
    if (!c->slabs.empty()) {
      Slab& s = c->slabs.back();
      if (s.ptr && s.used + padded <= s.bytes) {
        b.ptr = static_cast<char*>(s.ptr) + s.used;
        b.bytes = padded;
        b.slab = int(c->slabs.size());
        s.used += padded;
        ++s.live;
        c->arenaUsed += padded;
        *out = b.ptr;
        return UBR_OK;
      }
    }
    ubr_status st = devAlloc(c, b, grown, grown >= kDirectBytes);
    if (st != UBR_OK) return st;
  }
  *out = b.ptr;
  return UBR_OK;
}

// A context's first frame grows some thirty scratch blocks: 2-3 us each from
// the pool, 65 us whenever it has to grow (by 32 MB at least) and 0.8 us per MB;
// the slab is one cudaMalloc, worth it from about two growths on (first GI
// frames: 640x480 pt1 791 -> 726 us, 955x198 pt1 700 -> 598).
void scratchReserve(Context* c, size_t bytes) {
  if (c->arenaCap != 0 || bytes < (size_t(48) << 20) || bytes > kSlabBytes) return;
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  // a slab nothing was cut from serves no one any more
  if (!c->slabs.empty() && c->slabs.back().ptr && c->slabs.back().live == 0) {
    cudaFree(c->slabs.back().ptr);
    c->slabs.back() = Slab{};
  }
  c->slabs.push_back(Slab{p, bytes, 0, 0});
}

ubr_status workspaceMin(Context* c, void** out, size_t* bytes) {
  if (!c->workMin) UBR_CUDA(c, cudaMalloc(&c->workMin, kWorkspaceMin));
  *out = c->workMin;
  *bytes = kWorkspaceMin;
  return UBR_OK;
}

ubr_status workspaceGet(Context* c, int slot, size_t least, void** out, size_t* bytes) {
  if (c->arenaCap == 0) {
    if (scratchGet(c, slot, *bytes, out) == UBR_OK) return UBR_OK;
    cudaGetLastError();
  }
  const DevBuf* lend = nullptr;
  for (int k = 16; k <= 31 && size_t(k) < c->scratch.size(); ++k)
    if (c->scratch[size_t(k)].ptr && (!lend || c->scratch[size_t(k)].bytes > lend->bytes)) lend = &c->scratch[size_t(k)];
  if (lend && lend->bytes >= std::max(least, kWorkspaceMin)) {
    *out = lend->ptr;
    *bytes = std::min(*bytes, lend->bytes);
    return UBR_OK;
  }
  if (least <= kWorkspaceMin) {
    const size_t want = *bytes;
    const ubr_status st = workspaceMin(c, out, bytes);
    *bytes = std::min(*bytes, std::max(want, least));
    return st;
  }
  *bytes = least;
  return scratchGet(c, slot, least, out);
}

}  // namespace ubr

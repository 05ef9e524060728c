// ubr_context.h -- context, device buffers and scene object of libubr.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include "frame_planes.h"
#include "gi.cuh"
#include "ubr_internal.h"

namespace ubr {

// A device allocation owned by the context or a scene.  Grows on demand;
// contents are not preserved across growth.
struct DevBuf {
  void* ptr = nullptr;
  size_t bytes = 0;
  bool direct = false;  // from cudaMalloc, not from the context's pool
  bool slab = false;    // cut from the context's slab
  uint64_t call = 0;    // scratch: the call that asked for it last
};

// One cudaMalloc that a frame's large scratch blocks are cut from
// (scratchReserve); given back with the last of them.
struct Slab {
  void* ptr = nullptr;
  size_t bytes = 0;
  std::vector<std::pair<size_t, size_t>> free;  // (offset, bytes) by offset, neighbours merged
};

struct Context {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool ownStream = false;
  uint64_t arenaCap = 0;     // 0 = unlimited
  int leafMax = 1;           // wide-BVH leaf size (1..kWideLeafMax); 1 measured fastest
  int builder = 1;           // binary tree before the 8-wide collapse: 1 Karras radix tree, 2 PLOC
  int collapse = 0;          // 8-wide collapse: 0 library default, 1 greedy (fixed leaf size), 2 SAH-optimal (leaves 1..3)
  float sahPrimScale = 1.0f; // SAH collapse: weight of primitive tests against node visits
  int traceMode = 0;         // occlusion kernel: 0 chosen per launch, else the context desc's trace_mode
  uint64_t arenaUsed = 0;
  std::string lastError;
  // frame scratch, reused across frames
  std::vector<DevBuf> scratch;
  Slab slab;
  uint64_t call = 0;         // number of the running call (scratch blocks it uses carry it)
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  std::vector<cudaEvent_t> pev;  // profiling events, created on first use
  void* pinned = nullptr;    // small pinned host block for counters
  bool useGraphs = true;     // replay single-layer frames from a CUDA graph
  cudaGraphExec_t graphExec = nullptr;
  std::vector<unsigned char> graphKey;  // launch parameters the graph was captured with
  std::vector<void*> sceneHandles;      // live ubr_scene handles built on this context
  cudaMemPool_t pool = nullptr;         // stream-ordered device allocations (scenes, scratch)
  void* noallocArray = nullptr;         // device address of the allocation-free query's fixed array
  cudaEvent_t giEv[7] = {};             // GI pass stage boundaries, created on first use
};

struct Scene {
  Context* ctx = nullptr;
  DScene view;
  std::vector<DevBuf> bufs;  // owned allocations
  uint64_t primCount[4] = {0, 0, 0, 0};
  uint64_t nodes = 0;
  bool opaque = true;        // every primitive fully opaque: frames are one layer deep
  bool aoReceivers = false;  // a mesh or a non-outline primitive exists (coarse AO grid eligible)
  bool principled = false;   // some material uses the principled model
  // pt2 GI: a first hit can own a traced reflection (POV reflection > 0, or a
  // principled specular lobe); some can be glossy (a highlight-bearing POV
  // finish, or principled roughness^2 >= 0.015); an anisotropic principled
  // sphere / cylinder exists; the emissive primitives sampled as lights
  bool reflective = false, glossy = false, anisoPrincipled = false;
  EmitD emit;
  uint64_t deviceBytes = 0;
  double buildMs = 0.0;
  double flattenMs = 0.0;    // host: validation, primID ordering, chaining, material table
  double uploadMs = 0.0;     // host: allocations and copies queued
  float lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
};

// error helpers
ubr_status setError(Context* c, ubr_status s, const std::string& msg);
ubr_status cudaFail(Context* c, cudaError_t e, const char* what);
// allocate `bytes` on the context's device, honouring the arena cap
// (direct: by cudaMalloc instead of from the context's pool)
ubr_status devAlloc(Context* c, DevBuf& b, size_t bytes, bool direct = false);
void devFree(Context* c, DevBuf& b);
// scratch slot `i` of at least `bytes` (a quarter more when it grows, unless
// `slack` is false)
ubr_status scratchGet(Context* c, int i, size_t bytes, void** out, bool slack = true);

// Memory for the scratch blocks of a frame, before it asks for them: one
// allocation for the large blocks of the plan that have to grow, instead of one
// each.  The blocks of the last such allocation that this call
// has not asked for are given back first, so a context holds one at a time.
// None under an arena cap, for little, above kSlabBytes, or when it fails.
struct ScratchNeed {
  int slot;
  size_t bytes;
  bool slack = true;  // as scratchGet's
};
void scratchReserve(Context* c, const std::vector<ScratchNeed>& plan);
constexpr size_t kSlabBytes = size_t(512) << 20, kSlabLeast = size_t(48) << 20, kSlabBlock = size_t(1) << 16;

// Whether the arena cap leaves `bytes` (always without a cap).
bool arenaHolds(const Context* c, size_t bytes);

// A workspace of a pass that runs in chunks.  *bytes: what it uses well on
// entry, what it got on exit (at least `least`).  Scratch slot `slot`: all it
// wants, or what the arena cap leaves; where that is little or the allocation
// fails, memory that the context holds already, a block the running call does
// not use or what it lends (`lent`, may be null); else `least`, if the cap holds
// that.  A workspace does not stand in the way of other calls: where the cap
// would refuse an allocation, scratch that the running call has not asked for is
// released first.
constexpr int kGatherSlot = 149, kAdjointSlot = 150;
ubr_status workspaceGet(Context* c, int slot, size_t least, void* lent, size_t lentBytes, void** out, size_t* bytes);
// The running call has queued its last work on this block: other calls of this
// one's allocations may release it (ordered after that work).
void scratchDone(Context* c, int slot);

// typed view of scratch slot `slot` (count elements); a no-op once st != OK
template <class T>
T* scratchT(Context* c, int slot, size_t count, ubr_status& st) {
  void* ptr = nullptr;
  if (st == UBR_OK) st = scratchGet(c, slot, count * sizeof(T) + 16, &ptr);
  return static_cast<T*>(ptr);
}

// The allocation on `device` that holds the address, as the driver knows it;
// false for other memory.
bool deviceRange(int device, const void* ptr, uintptr_t& start, size_t& size);
// Whether [ptr, ptr + bytes) lies within one allocation on the device.  Kernels
// write a caller's memory only where this holds: a copy or memset checks what
// it is given and fails with an error, a kernel's store faults.  One object per
// call: it asks the driver once per allocation.
struct DeviceMemory {
  explicit DeviceMemory(int device) : device(device) {}
  bool operator()(const void* ptr, size_t bytes) {
    return known(ptr, bytes, [&](uintptr_t& start, size_t& size) { return deviceRange(device, ptr, start, size); });
  }
  int device;
  KnownRanges known;
};

// Frame parameters and light table of a render description (camera basis,
// lights, AO / fog / gamma settings), validated.
ubr_status makeParams(Context* c, const ubr_render_desc& d, Params& p, std::vector<LightD>& lights);

#define UBR_CUDA(ctx, call)                                  \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return cudaFail((ctx), e_, #call); \
  } while (0)

}  // namespace ubr

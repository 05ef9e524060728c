// A context's device memory (csrc/context.cu) on a fake CUDA runtime that keeps
// a list of the live allocations: what is held, what is given back, and that
// no two blocks share memory.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "ubr_context.h"

using namespace ubr;

namespace fake {
std::map<uintptr_t, size_t> live;  // address -> bytes
uintptr_t next = uintptr_t(1) << 32;
size_t held = 0, peak = 0, limit = ~size_t(0);
int calls = 0;
cudaError_t take(void** p, size_t n) {
  ++calls;
  if (held + n > limit) return cudaErrorMemoryAllocation;
  next = (next + 511) & ~uintptr_t(511);
  *p = reinterpret_cast<void*>(next);
  live[next] = n;
  next += n;
  held += n;
  peak = held > peak ? held : peak;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  auto it = live.find(reinterpret_cast<uintptr_t>(p));
  if (it == live.end()) {
    std::printf("FAILED: freed an address that is not allocated\n");
    std::exit(1);
  }
  held -= it->second;
  live.erase(it);
  return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::take(p, n); }
cudaError_t cudaFree(void* p) { return fake::give(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::take(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::give(p); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok && ++failures < 20) std::printf("FAILED: %s\n", what);
}

// Every scratch block lies within one live allocation, no two meet, and the
// context's count of its memory is theirs.
static void consistent(const Context& c) {
  size_t sum = 0;
  std::map<uintptr_t, size_t> by;
  for (const DevBuf& b : c.scratch) {
    if (!b.ptr) continue;
    sum += b.bytes;
    const uintptr_t at = reinterpret_cast<uintptr_t>(b.ptr);
    auto it = fake::live.upper_bound(at);
    check(it != fake::live.begin(), "a block lies in a live allocation");
    if (it == fake::live.begin()) continue;
    --it;
    check(at + b.bytes <= it->first + it->second, "a block lies within its allocation");
    check(by.emplace(at, b.bytes).second, "no two blocks start together");
  }
  uintptr_t end = 0;
  for (const auto& [at, n] : by) {
    check(at >= end, "no two blocks meet");
    end = at + n;
  }
  check(c.arenaUsed == sum, "the arena counts the blocks");
}

static Context& fresh(uint64_t cap) {
  static Context* c = nullptr;
  delete c;
  c = new Context();
  c->arenaCap = cap;
  c->pool = reinterpret_cast<cudaMemPool_t>(16);
  fake::live.clear();
  fake::held = fake::peak = 0;
  fake::limit = ~size_t(0);
  return *c;
}

static size_t blocks(const Context& c) {
  size_t n = 0;
  for (const DevBuf& b : c.scratch) n += b.ptr ? b.bytes : 0;
  return n;
}

#include "context_memory_cases.hpp"

int main() {
  cases();
  if (failures) std::printf("%d failures\n", failures);
  return failures ? 1 : 0;
}

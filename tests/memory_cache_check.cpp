// The memory kept between calls (sih26_b200/csrc/device_cache.cuh) against a fake of the CUDA runtime that
// counts what is allocated, gives the same addresses again after a reset, and names contexts as the driver
// does. Prints ok, or the first expectation that fails; run by tests/test_memory_cache_cpu.py.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "device_cache.cuh"

static unsigned long long g_context = 1;  // 0: the driver does not say
static std::set<void*> g_live;            // the present context's allocations
static int g_bad_frees = 0, g_allocations = 0, g_fail_next = 0;
static unsigned long long g_next = 0x1000000;

static void reset() {  // cudaDeviceReset: the memory goes, addresses start again
  g_live.clear();
  g_next = 0x1000000;
  ++g_context;
}
static cudaError_t give(void** p, size_t bytes) {
  if (g_fail_next > 0) {
    --g_fail_next;
    return cudaErrorMemoryAllocation;
  }
  *p = reinterpret_cast<void*>(g_next);
  g_next += (bytes + 255) & ~size_t(255);
  g_live.insert(*p);
  ++g_allocations;
  return cudaSuccess;
}
static cudaError_t drop(void* p) {
  if (g_live.erase(p) == 0) ++g_bad_frees;
  return cudaSuccess;
}
static CUresult fake_id(CUcontext, unsigned long long* id) {
  *id = g_context;
  return g_context ? CUDA_SUCCESS : CUDA_ERROR_INVALID_CONTEXT;
}

extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t bytes) { return give(p, bytes); }
cudaError_t CUDARTAPI cudaFree(void* p) { return drop(p); }
cudaError_t CUDARTAPI cudaMallocHost(void** p, size_t bytes) { return give(p, bytes); }
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t bytes, unsigned) { return give(p, bytes); }
cudaError_t CUDARTAPI cudaFreeHost(void* p) { return drop(p); }
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned int, unsigned long long,
                                                       cudaDriverEntryPointQueryResult* r) {
  *f = reinterpret_cast<void*>(&fake_id);
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

#define WANT(x)                                      \
  do {                                               \
    if (!(x)) {                                      \
      std::printf("line %d: %s\n", __LINE__, #x);    \
      return 1;                                      \
    }                                                \
  } while (0)

int main() {
  using sih26::Chunk;
  sih26::MemoryCache& mc = sih26::MemoryCache::get();
  // kept and handed out again, to one owner at a time, not to a request of under half its size
  const Chunk a = mc.take_device(0, 1000);
  mc.give_device(a);
  WANT(mc.kept(0) == 1000 && mc.take_device(0, 400).p != a.p);
  const Chunk b = mc.take_device(0, 900);
  WANT(b.p == a.p && b.bytes == 1000 && mc.take_device(0, 900).p != a.p);
  mc.give_device(b);
  const Chunk h = mc.take_pinned(500);
  mc.give_pinned(h);
  // a reset: the chunks kept are forgotten, and what now lives at their addresses is left alone
  reset();
  WANT(mc.kept(0) == 0);
  void *other[2] = {nullptr, nullptr};
  WANT(give(&other[0], 1000) == cudaSuccess && give(&other[1], 1000) == cudaSuccess);
  const Chunk c = mc.take_device(0, 1000), g = mc.take_pinned(500);
  WANT(c.p != other[0] && c.p != other[1] && g.p != other[0] && g.p != other[1]);
  WANT(g_live.count(c.p) && g_live.count(g.p));
  // a chunk that was out when its context ended is not kept and not freed
  reset();
  WANT(give(&other[0], 1000) == cudaSuccess && other[0] == reinterpret_cast<void*>(0x1000000));
  mc.give_device(b);
  mc.give_pinned(g);
  WANT(mc.kept(0) == 0 && g_live.count(other[0]) && g_bad_frees == 0);
  // an allocation that fails gives what is kept back and tries again
  mc.give_device(mc.take_device(0, 4096));
  WANT(mc.kept(0) == 4096);
  g_fail_next = 1;
  const size_t live = g_live.size();
  WANT(mc.take_device(0, 100000).p != nullptr && mc.kept(0) == 0 && g_live.size() == live);
  // on request
  mc.give_device(mc.take_device(0, 4096));
  mc.give_pinned(mc.take_pinned(4096));
  const size_t before = g_live.size();
  WANT(mc.release(0) == 4096 && g_live.size() == before - 2 && mc.release(0) == 0);
  // the bound
  const Chunk big = mc.take_device(0, sih26::MemoryCache::kKeepDevice), more = mc.take_device(0, 1);
  mc.give_device(big);
  mc.give_device(more);
  WANT(mc.kept(0) == sih26::MemoryCache::kKeepDevice && !g_live.count(more.p));
  // no context id: nothing is kept, everything is freed
  mc.release(0);
  g_context = 0;
  const Chunk u = mc.take_device(0, 64);
  mc.give_device(u);
  WANT(!g_live.count(u.p) && g_bad_frees == 0);
  std::puts("ok");
  return 0;
}

// Device memory and pinned read-back buffers kept between calls.
//
// Every entry point takes its workspace from a stream-ordered pool and frees
// it before it returns.  The device's default pool gives unused memory back
// to the driver at the next synchronisation, which each entry point performs,
// so every call mapped its workspace anew: 0.44 ms of the 0.74 ms that an LU
// of n = 100 took, 0.75 ms of an n = 1024 one, and under a server's seven
// threads, whose mappings serialise, more time than the factorisations.  The
// two pools here (workspaces, and factors that outlive a call) keep up to
// kKeep bytes of unused memory each; more than that goes back at the next
// synchronisation, and dp_memory_trim or the end of a server gives back the
// rest.  Another allocation of the process that runs short gets it without that
// (2.3 GiB kept, the device otherwise full: a cudaMalloc of 1 GiB more than its
// free memory succeeded).  An allocation that fails is tried once more after a trim.  The pools
// are the driver's own, safe for any mix of threads and streams; a block
// freed on one stream is handed to another only once the free has been
// reached (no waits between streams are inserted for it).
#include <mutex>

#include "delayed_pivoting_b200.h"
#include "dp_device.cuh"
#include "dp_kernels.h"

namespace dp {
namespace {

constexpr int kMaxDevices = 64;
// bytes of unused memory kept: workspaces of an n = 32768 LU (0.6 GB) and
// the factors of one of n = 16384 (2.2 GB) stay; both are small beside the
// device's 180 GB
constexpr unsigned long long kKeep[2] = {1ull << 30, 3ull << 30};

std::mutex g_mutex;
cudaMemPool_t g_pools[kMaxDevices][2] = {};

cudaMemPool_t pool_of(int dev, int kind) {
  std::lock_guard<std::mutex> lock(g_mutex);
  cudaMemPool_t& p = g_pools[dev][kind];
  if (!p) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t fresh = nullptr;
    if (cudaMemPoolCreate(&fresh, &props) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    unsigned long long keep = kKeep[kind];
    int off = 0;
    cudaMemPoolSetAttribute(fresh, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(fresh, cudaMemPoolReuseAllowInternalDependencies, &off);
    p = fresh;
  }
  return p;
}

void trim(int dev) {
  std::lock_guard<std::mutex> lock(g_mutex);
  for (cudaMemPool_t p : g_pools[dev])
    if (p) cudaMemPoolTrimTo(p, 0);
}

cudaError_t alloc(void** out, size_t bytes, cudaStream_t st, int kind) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaMemPool_t p = dev >= 0 && dev < kMaxDevices ? pool_of(dev, kind) : nullptr;
  if (!p) return cudaMallocAsync(out, bytes, st);
  e = cudaMallocFromPoolAsync(out, bytes, p, st);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim(dev);
    e = cudaMallocFromPoolAsync(out, bytes, p, st);
  }
  return e;
}

// One pinned block per host thread (device-to-host copies into pageable
// memory go through the driver's own staging buffer and cost about 5 us more
// each); freed when the thread ends.
struct Pinned {
  void* p = nullptr;
  ~Pinned() {
    if (p) cudaFreeHost(p);
  }
};
thread_local Pinned g_pinned;

}  // namespace

cudaError_t workspace_alloc(void** out, size_t bytes, cudaStream_t st) {
  return alloc(out, bytes, st, 0);
}
cudaError_t resident_alloc(void** out, size_t bytes, cudaStream_t st) {
  return alloc(out, bytes, st, 1);
}

void memory_trim() {
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) trim(dev);
}

void* pinned_stage(size_t bytes) {
  if (bytes > kPinnedStageBytes) return nullptr;
  if (!g_pinned.p &&
      cudaHostAlloc(&g_pinned.p, kPinnedStageBytes, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_pinned.p = nullptr;
  }
  return g_pinned.p;
}

}  // namespace dp

extern "C" int dp_memory_trim(void) {
  dp::memory_trim();
  return DP_SUCCESS;
}

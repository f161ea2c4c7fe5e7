// Device scratch of single calls, and the counters' buffers: stream-ordered
// allocations from a memory pool of the library's own, one per device.  A call allocates on its stream
// and gives the memory back on it, so calls on any streams and threads share
// the pool safely, and a captured call's allocations become part of its
// graph.  The pool keeps up to kKeep bytes between calls (a pool that keeps
// nothing maps the memory anew after every synchronisation, about 0.8 ms a
// call) and gives everything back when the device's last database or counter
// set is closed, or when the library needs it for something else (device_alloc).
#include <cuda_runtime.h>

#include <mutex>

#include "k2g_internal.h"

namespace k2g {
namespace {

constexpr uint64_t kKeep = 1ull << 30;

struct Pool {
  std::mutex mu;
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;   // for memory that no call's stream owns
  int users = 0;               // open databases and counter sets
};
Pool g_pools[64];

}  // namespace

cudaError_t scratch_alloc(void **p, size_t bytes, int device, cudaStream_t st) {
  Pool &d = g_pools[device & 63];
  {
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.pool) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.handleTypes = cudaMemHandleTypeNone;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      cudaError_t e = cudaMemPoolCreate(&d.pool, &props);
      if (e != cudaSuccess) {
        d.pool = nullptr;
        return e;
      }
      uint64_t keep = kKeep;
      e = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaMallocFromPoolAsync(p, bytes ? bytes : 1, d.pool, st);
}

cudaError_t scratch_alloc_now(void **p, size_t bytes, int device) {
  Pool &d = g_pools[device & 63];
  {
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.st) {
      const cudaError_t e = cudaStreamCreateWithFlags(&d.st, cudaStreamNonBlocking);
      if (e != cudaSuccess) return e;
    }
  }
  cudaError_t e = scratch_alloc(p, bytes, device, d.st);
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(d.st);
  if (e != cudaSuccess) {
    cudaFreeAsync(*p, d.st);
    *p = nullptr;
  }
  return e;
}

void scratch_free_now(void *p, int device) {
  if (p) cudaFreeAsync(p, g_pools[device & 63].st);
}

cudaError_t device_alloc(void **p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes);
  int device = 0;
  if (e != cudaErrorMemoryAllocation || cudaGetDevice(&device) != cudaSuccess) return e;
  Pool &d = g_pools[device & 63];
  {
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.pool) return e;
    // (what was given back on a stream counts once its end has been waited for)
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemPoolTrimTo(d.pool, 0) != cudaSuccess) return e;
  }
  (void)cudaGetLastError();
  return cudaMalloc(p, bytes);
}

void scratch_opened(int device) {
  Pool &d = g_pools[device & 63];
  std::lock_guard<std::mutex> lock(d.mu);
  d.users++;
}

void scratch_closed(int device) {
  Pool &d = g_pools[device & 63];
  std::lock_guard<std::mutex> lock(d.mu);
  if (--d.users == 0 && d.pool) {
    if (d.st) cudaStreamSynchronize(d.st);
    cudaMemPoolTrimTo(d.pool, 0);
  }
}

}  // namespace k2g

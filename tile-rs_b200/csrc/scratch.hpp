// Device scratch of the operators: taken on the caller's stream when a call needs it, returned on that stream when its last kernel
// is queued, from a memory pool of the library's own on each device.  The device's default pool belongs to the host program and
// is neither used nor changed.
//
// The pool keeps what is returned to it (no trimming at synchronisation points, so that from the second call on taking and
// returning are bookkeeping on the stream), up to one sixteenth of the device's memory; closing the last handle of a device
// gives all of it back.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>

namespace tsm100 {
namespace scratch {

struct Pools {
  std::mutex mu;
  std::map<int, cudaMemPool_t> of_device;
};
inline Pools& pools() {
  static Pools p;
  return p;
}

inline cudaError_t current_pool(cudaMemPool_t* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Pools& p = pools();
  std::lock_guard<std::mutex> lock(p.mu);
  auto it = p.of_device.find(dev);
  if (it != p.of_device.end()) {
    *out = it->second;
    return cudaSuccess;
  }
  // the first call may come while this thread captures a stream; nothing here belongs into the graph
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  e = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return e;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  e = cudaMemPoolCreate(&pool, &props);
  size_t free_bytes = 0, total = 0;
  if (e == cudaSuccess) e = cudaMemGetInfo(&free_bytes, &total);
  uint64_t keep = total / 16;
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  if (e != cudaSuccess && pool) cudaMemPoolDestroy(pool);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return e;
  p.of_device[dev] = pool;
  *out = pool;
  return cudaSuccess;
}

// A build may cap what one call takes (in bytes); calls that would need more take the form that needs none.
#ifdef TSM100_SCRATCH_LIMIT
constexpr size_t kLimit = TSM100_SCRATCH_LIMIT;
#else
constexpr size_t kLimit = SIZE_MAX;
#endif

inline cudaError_t take(void** out, size_t bytes, cudaStream_t s) {
  if (bytes > kLimit) return cudaErrorMemoryAllocation;
  cudaMemPool_t pool;
  const cudaError_t e = current_pool(&pool);
  return e != cudaSuccess ? e : cudaMallocFromPoolAsync(out, bytes, pool, s);
}

// What no call has in use any more goes back to the device.
inline void give_back(int dev) {
  Pools& p = pools();
  std::lock_guard<std::mutex> lock(p.mu);
  auto it = p.of_device.find(dev);
  if (it != p.of_device.end() && cudaMemPoolTrimTo(it->second, 0) != cudaSuccess) (void)cudaGetLastError();
}

}  // namespace scratch
}  // namespace tsm100

// pool.cpp — device memory, pinned host memory and streams behind the
// handles.
//
// A model's life used to be driver calls: cudaMalloc 0.36 ms and cudaFree
// 0.29 ms for each of its dozen buffers, cudaMallocHost 1.9 ms, a stream
// 0.05 ms — 6.5 ms of a 7 ms factor-and-predict at n = 1024.  Here:
//
//  * device buffers up to POOL_MAX_BLOCK come from one CUDA memory pool per
//    device (3 µs).  An allocation is ordered on a private stream that is
//    drained before the pointer is returned, so any stream may use it at once;
//    a free first waits for the device, as cudaFree does.  The pool gives
//    memory above POOL_KEEP back to the driver whenever it is drained, and all
//    of its unused memory when an allocation fails.
//  * pinned blocks and idle streams are kept in small bounded lists (PINNED_KEEP
//    bytes, STREAM_KEEP streams of a kind); what does not fit is freed.
//
// Every list is behind one mutex.  Buffers keep their device, so they may be
// freed with any device current.  The lists live until the process ends.

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <vector>

#include "pool.h"

namespace gprx {

namespace {

constexpr size_t POOL_KEEP = (size_t)1 << 30;
constexpr size_t POOL_MAX_BLOCK = (size_t)256 << 20;  // larger buffers go to cudaMalloc
constexpr size_t PINNED_KEEP = (size_t)8 << 20;
constexpr size_t PINNED_MAX_BLOCK = (size_t)1 << 20;
constexpr size_t STREAM_KEEP = 16;

struct DevicePool {
  bool tried = false;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
  std::vector<cudaStream_t> idle[2];  // by priority: normal, high
};

struct Pools {
  std::mutex mu;
  std::map<int, DevicePool> dev;
  std::map<size_t, std::vector<void*>> pinned;  // by size class
  size_t pinned_bytes = 0;
};

Pools& pools() {
  static Pools* p = new Pools;  // never destroyed: handles may outlive static objects
  return *p;
}

size_t pinned_class(size_t bytes) {
  size_t c = 4096;
  while (c < bytes) c *= 2;
  return c;
}

// The device's pool, made at its first use; null when the device has none.
DevicePool* device_pool(Pools& p, int device) {
  DevicePool& d = p.dev[device];
  if (!d.tried) {
    d.tried = true;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    unsigned long long keep = POOL_KEEP;
    if (cudaMemPoolCreate(&d.pool, &props) != cudaSuccess) d.pool = nullptr;
    if (d.pool && (cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                   cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking) != cudaSuccess)) {
      cudaMemPoolDestroy(d.pool);
      d.pool = nullptr;
    }
    if (!d.pool) (void)cudaGetLastError();
  }
  return d.pool ? &d : nullptr;
}

}  // namespace

cudaError_t device_alloc(void** out, size_t bytes, int* device) {
  *out = nullptr;
  cudaError_t e = cudaGetDevice(device);
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (DevicePool* d = device_pool(p, *device)) {
      pool = d->pool;
      stream = d->stream;
    }
  }
  if (pool && bytes <= POOL_MAX_BLOCK) {
    for (int attempt = 0; attempt < 2; ++attempt) {
      e = cudaMallocFromPoolAsync(out, bytes, pool, stream);
      if (e == cudaSuccess) return cudaStreamSynchronize(stream);
      (void)cudaGetLastError();
      *out = nullptr;
      if (attempt == 0) {
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(pool, 0);
      }
    }
    return e;
  }
  e = cudaMalloc(out, bytes);
  if (e == cudaErrorMemoryAllocation && pool) {
    (void)cudaGetLastError();
    cudaDeviceSynchronize();
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMalloc(out, bytes);
  }
  if (e != cudaSuccess) *out = nullptr;
  return e;
}

void device_free(void* ptr, size_t bytes, int device) {
  if (!ptr) return;
  cudaStream_t stream = nullptr;
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (DevicePool* d = device_pool(p, device)) stream = d->stream;
  }
  if (!stream || bytes > POOL_MAX_BLOCK) {
    cudaFree(ptr);
    return;
  }
  int was = device;
  cudaGetDevice(&was);
  if (was != device) cudaSetDevice(device);
  // a wait that was refused (a capture elsewhere) leaves it to cudaFree's own
  if (cudaDeviceSynchronize() == cudaSuccess) cudaFreeAsync(ptr, stream);
  else cudaFree(ptr);
  if (was != device) cudaSetDevice(was);
}

cudaError_t pinned_alloc(void** out, size_t bytes) {
  *out = nullptr;
  const size_t c = pinned_class(bytes);
  if (c > PINNED_MAX_BLOCK) return cudaMallocHost(out, bytes);
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    auto& list = p.pinned[c];
    if (!list.empty()) {
      *out = list.back();
      list.pop_back();
      p.pinned_bytes -= c;
      return cudaSuccess;
    }
  }
  return cudaMallocHost(out, c);
}

void pinned_free(void* ptr, size_t bytes) {
  if (!ptr) return;
  const size_t c = pinned_class(bytes);
  if (c <= PINNED_MAX_BLOCK) {
    cudaDeviceSynchronize();  // cudaFreeHost's wait: no copy into the block is in flight
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (p.pinned_bytes + c <= PINNED_KEEP) {
      p.pinned[c].push_back(ptr);
      p.pinned_bytes += c;
      return;
    }
  }
  cudaFreeHost(ptr);
}

cudaError_t stream_acquire(cudaStream_t* out, bool high) {
  *out = nullptr;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    auto& list = p.dev[device].idle[high ? 1 : 0];
    if (!list.empty()) {
      *out = list.back();
      list.pop_back();
      return cudaSuccess;
    }
  }
  if (!high) return cudaStreamCreateWithFlags(out, cudaStreamNonBlocking);
  int lo = 0, hi = 0;
  if ((e = cudaDeviceGetStreamPriorityRange(&lo, &hi)) != cudaSuccess) return e;
  return cudaStreamCreateWithPriority(out, cudaStreamNonBlocking, hi);
}

void stream_release(cudaStream_t s, bool high, int device) {
  if (!s) return;
  if (cudaStreamSynchronize(s) == cudaSuccess) {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    auto& list = p.dev[device].idle[high ? 1 : 0];
    if (list.size() < STREAM_KEEP) {
      list.push_back(s);
      return;
    }
  }
  cudaStreamDestroy(s);
}

}  // namespace gprx

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
//    a free first waits for its owner's streams (Lane) and drains it again: then
//    the pool gives what it holds above POOL_KEEP back to the driver.  All of its
//    unused memory goes back when an allocation fails.
//  * an online model's second factor-sized buffer waits here between deletes
//    (spare_keep), so that it is there for the next one and for nobody's loss: all
//    of them hold SPARE_KEEP at most, and an allocation that would fail takes them.
//  * pinned blocks and idle streams are kept in small bounded lists (PINNED_KEEP
//    bytes, STREAM_KEEP streams of a kind); what does not fit is freed.
//
// Nothing here waits for the whole device: that is an error while any stream is
// being captured (a batched fit's rounds on another thread, a caller's graph)
// and ends the capture with an error of its own.
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
constexpr size_t SPARE_KEEP = (size_t)4 << 30;
constexpr size_t PINNED_KEEP = (size_t)8 << 20;
constexpr size_t STREAM_KEEP = 16;

struct DevicePool {
  bool tried = false;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
  std::vector<cudaStream_t> idle[2];  // by priority: normal, high
};

struct SpareBlock {
  void* ptr;
  size_t bytes;
  int device;
};

struct Pools {
  std::mutex mu;
  std::map<int, DevicePool> dev;
  std::map<const void*, SpareBlock> spare;  // by owner
  size_t spare_bytes = 0;
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

// Frees a block that nothing uses.
void free_idle(void* ptr, size_t bytes, int device) {
  if (!ptr) return;
  cudaStream_t stream = nullptr;
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (DevicePool* d = device_pool(p, device)) stream = d->stream;
  }
  cudaError_t e;
  if (!stream || bytes > POOL_MAX_BLOCK) e = cudaFree(ptr);
  else if ((e = cudaFreeAsync(ptr, stream)) == cudaSuccess)
    e = cudaStreamSynchronize(stream);  // what the pool holds past POOL_KEEP goes to the driver
  if (e != cudaSuccess) (void)cudaGetLastError();
}

// Removes the owner's spare block (of any owner with null; on `device` only unless −1)
// from the list; ptr is null when there is none.
SpareBlock spare_remove(const void* owner, int device) {
  Pools& p = pools();
  std::lock_guard<std::mutex> lock(p.mu);
  for (auto it = owner ? p.spare.find(owner) : p.spare.begin(); it != p.spare.end(); ++it) {
    if (device >= 0 && it->second.device != device) {
      if (owner) break;
      continue;
    }
    const SpareBlock b = it->second;
    p.spare_bytes -= b.bytes;
    p.spare.erase(it);
    return b;
  }
  return {nullptr, 0, 0};
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
  const bool pooled = pool && bytes <= POOL_MAX_BLOCK;
  for (int attempt = 0; attempt < 2; ++attempt) {
    e = pooled ? cudaMallocFromPoolAsync(out, bytes, pool, stream) : cudaMalloc(out, bytes);
    if (e == cudaSuccess) return pooled ? cudaStreamSynchronize(stream) : e;
    (void)cudaGetLastError();
    *out = nullptr;
    if (e != cudaErrorMemoryAllocation) break;
    // the spares, and what the pool holds unused, go back to the driver
    for (SpareBlock b; (b = spare_remove(nullptr, *device)).ptr;) free_idle(b.ptr, b.bytes, b.device);
    if (!pool) continue;
    cudaStreamSynchronize(stream);
    cudaMemPoolTrimTo(pool, 0);
  }
  return e;
}

void device_free(void* ptr, size_t bytes, int device, const Lane& lane) {
  // work that may use it could not be waited for: nobody else gets it
  if (ptr && (lane.drain() || bytes > POOL_MAX_BLOCK)) free_idle(ptr, bytes, device);
}

void spare_keep(const void* owner, void* ptr, size_t bytes, int device) {
  if (!ptr) return;
  spare_drop(owner);
  {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (p.spare_bytes + bytes <= SPARE_KEEP) {
      p.spare[owner] = {ptr, bytes, device};
      p.spare_bytes += bytes;
      return;
    }
  }
  free_idle(ptr, bytes, device);
}

void* spare_take(const void* owner, size_t* bytes, int* device) {
  const SpareBlock b = spare_remove(owner, -1);
  if (!b.ptr) return nullptr;
  if (b.bytes < *bytes) {
    free_idle(b.ptr, b.bytes, b.device);
    return nullptr;
  }
  *bytes = b.bytes;
  *device = b.device;
  return b.ptr;
}

void spare_drop(const void* owner) {
  const SpareBlock b = spare_remove(owner, -1);
  free_idle(b.ptr, b.bytes, b.device);
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

void pinned_free(void* ptr, size_t bytes, const Lane& lane) {
  if (!ptr) return;
  const size_t c = pinned_class(bytes);
  if (c <= PINNED_MAX_BLOCK && lane.drain()) {  // no copy into the block is in flight
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    if (p.pinned_bytes + c <= PINNED_KEEP) {
      p.pinned[c].push_back(ptr);
      p.pinned_bytes += c;
      return;
    }
  }
  if (cudaFreeHost(ptr) != cudaSuccess) (void)cudaGetLastError();
}

// A non-blocking stream of the current device, normal or highest priority.
static cudaError_t stream_acquire(cudaStream_t* out, bool high) {
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

// Back to the list; one that was not drained is given up.
static void stream_release(cudaStream_t s, bool high, int device, bool drained) {
  if (drained) {
    Pools& p = pools();
    std::lock_guard<std::mutex> lock(p.mu);
    auto& list = p.dev[device].idle[high ? 1 : 0];
    if (list.size() < STREAM_KEEP) {
      list.push_back(s);
      return;
    }
  }
  if (cudaStreamDestroy(s) != cudaSuccess) (void)cudaGetLastError();
}

cudaError_t Lane::open() {
  if (s_[0]) return cudaSuccess;
  cudaError_t e = cudaGetDevice(&device_);
  return e != cudaSuccess ? e : stream_acquire(&s_[0], false);
}

cudaError_t Lane::open_sides() {
  for (int i = 1; i < 3; ++i) {
    if (s_[i]) continue;
    const cudaError_t e = stream_acquire(&s_[i], true);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

bool Lane::drain() const {
  bool ok = true;
  for (cudaStream_t s : s_)
    if (s && cudaStreamSynchronize(s) != cudaSuccess) {
      (void)cudaGetLastError();
      ok = false;
    }
  return ok;
}

void Lane::close() {
  const bool drained = drain();
  for (int i = 0; i < 3; ++i) {
    if (s_[i]) stream_release(s_[i], i > 0, device_, drained);
    s_[i] = nullptr;
  }
}

}  // namespace gprx

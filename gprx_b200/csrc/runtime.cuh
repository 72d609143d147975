// runtime.cuh — host runtime shared by the handles: device buffers, the
// per-thread error record, status mapping.
#pragma once

#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "pool.h"

namespace gprx {

// Thread-local record behind gprx_last_error().
gprx_error_info& last_error();
gprx_status set_error(gprx_status st, const std::string& msg);
gprx_status set_cuda_error(cudaError_t e, const char* where);
gprx_status set_cholesky_error(double jitter, uint64_t size, int stage);

#define GPRX_CUDA_TRY(expr)                                   \
  do {                                                        \
    cudaError_t e_ = (expr);                                  \
    if (e_ != cudaSuccess) return ::gprx::set_cuda_error(e_, #expr); \
  } while (0)

// Owning device buffer of the owner with these streams.
template <typename T>
struct DevBuf {
  const Lane& lane;
  T* p = nullptr;
  size_t n = 0;
  int device = 0;
  explicit DevBuf(const Lane& l) : lane(l) {}
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { reset(); }
  cudaError_t alloc(size_t count) {
    reset();
    if (count == 0) return cudaSuccess;
    cudaError_t e = device_alloc((void**)&p, count * sizeof(T), &device);
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
  // grows (never shrinks); contents are not kept
  cudaError_t ensure(size_t count) { return count <= n ? cudaSuccess : alloc(count); }
  void reset() {
    device_free(p, n * sizeof(T), device, lane);
    p = nullptr;
    n = 0;
  }
  // alloc, in the owner's spare block (pool.h) where it is there and large enough
  cudaError_t take_spare(const void* owner, size_t count) {
    reset();
    size_t bytes = count * sizeof(T);
    p = static_cast<T*>(spare_take(owner, &bytes, &device));
    if (!p) return alloc(count);
    n = bytes / sizeof(T);
    return cudaSuccess;
  }
  // the buffer, whose work has been waited for, becomes the owner's spare block
  void keep_spare(const void* owner) {
    spare_keep(owner, p, n * sizeof(T), device);
    p = nullptr;
    n = 0;
  }
};

// Pinned host scratch.
template <typename T>
struct HostPinned {
  const Lane& lane;
  T* p = nullptr;
  size_t n = 0;
  explicit HostPinned(const Lane& l) : lane(l) {}
  HostPinned(const HostPinned&) = delete;
  HostPinned& operator=(const HostPinned&) = delete;
  ~HostPinned() { reset(); }
  cudaError_t ensure(size_t count) {
    if (count <= n) return cudaSuccess;
    reset();
    cudaError_t e = pinned_alloc((void**)&p, count * sizeof(T));
    if (e == cudaSuccess) n = count;
    return e;
  }
  void reset() {
    pinned_free(p, n * sizeof(T), lane);
    p = nullptr;
    n = 0;
  }
};

// Query points of a prediction whose results' pinned block (256 KB) stays with the
// handle; that of a larger call goes back to the shared list.
constexpr int PRED_KEEP = 16384;

inline long long round_ld(long long n) { return (n + 31) / 32 * 32; }

bool all_finite(const double* v, size_t n);

// Reads the device status word (after the stream drained) and maps it.
gprx_status status_to_error(const DevStatus& st, double jitter, uint64_t size, int stage);

}  // namespace gprx

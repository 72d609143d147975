// pool.h — see pool.cpp.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace gprx {

// The streams of one owner (a handle).  All work on the owner's buffers is
// ordered by them, so a buffer's release waits for them and for nothing else:
// no wait on the device, which a capture on any other stream would forbid.
class Lane {
 public:
  Lane() = default;
  Lane(const Lane&) = delete;
  Lane& operator=(const Lane&) = delete;
  ~Lane() { close(); }
  cudaError_t open();        // the main stream, on the current device
  cudaError_t open_sides();  // two of the highest priority
  // Waits for every stream; false when one cannot be waited for.
  bool drain() const;
  // Drains and gives the streams back; later releases have nothing to wait for.
  void close();
  cudaStream_t main() const { return s_[0]; }
  cudaStream_t aux() const { return s_[1]; }
  cudaStream_t aux2() const { return s_[2]; }

 private:
  int device_ = 0;
  cudaStream_t s_[3] = {nullptr, nullptr, nullptr};
};

// Device memory on the current device (*device receives it); usable from any
// stream on return.
cudaError_t device_alloc(void** out, size_t bytes, int* device);
void device_free(void* ptr, size_t bytes, int device, const Lane& lane);

// One spare block an owner: a buffer it will want again but can do without.  All
// spares of a device are freed before an allocation there fails, and what goes
// beyond SPARE_KEEP bytes in all is freed at once.
// Nothing uses the block any more: its owner has waited for its work.
void spare_keep(const void* owner, void* ptr, size_t bytes, int device);
// The owner's spare of at least *bytes (*bytes and *device receive its own), or null.
void* spare_take(const void* owner, size_t* bytes, int* device);
void spare_drop(const void* owner);

// Pinned host memory; pinned_free takes the size asked for and keeps blocks of at
// most PINNED_MAX_BLOCK bytes for reuse.
constexpr size_t PINNED_MAX_BLOCK = (size_t)1 << 20;
cudaError_t pinned_alloc(void** out, size_t bytes);
void pinned_free(void* ptr, size_t bytes, const Lane& lane);

}  // namespace gprx

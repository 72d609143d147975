// pool.h — see pool.cpp.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace gprx {

// Device memory on the current device (*device receives it); usable from any
// stream on return.  device_free waits for the device first.
cudaError_t device_alloc(void** out, size_t bytes, int* device);
void device_free(void* ptr, size_t bytes, int device);

// Pinned host memory; pinned_free takes the size asked for.
cudaError_t pinned_alloc(void** out, size_t bytes);
void pinned_free(void* ptr, size_t bytes);

// Non-blocking streams of the current device, normal or highest priority;
// stream_release drains the stream.
cudaError_t stream_acquire(cudaStream_t* out, bool high);
void stream_release(cudaStream_t s, bool high, int device);

}  // namespace gprx

// device_memory.cuh — device allocations of the library, and the scratch that calls without a
// context keep between them.
#pragma once

#include <cstddef>
#include <cuda_runtime_api.h>

namespace gwmb {

// Scratch of one call, ordered on stream s; freed with cudaFreeAsync.  It comes from a pool of
// the library per device that keeps up to 256 MB between calls (larger scratch goes back to the
// device at the next synchronisation): the default pool gives everything back at each call's
// end, and mapping it again cost more than the steps of a scalar transport.  Allocations are
// stream-ordered, so threads and streams share the pool safely.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);

// Gives back what the pools keep, on every device.
void trim_scratch();

// cudaMalloc and cudaMallocAsync, tried once more without the kept scratch when there is no
// room.  A failure leaves no error behind for the next launch to report.
cudaError_t device_alloc_bytes(void** p, size_t bytes);
cudaError_t device_alloc_async_bytes(void** p, size_t bytes, cudaStream_t s);
template <class T>
cudaError_t device_alloc(T** p, size_t bytes) {
  return device_alloc_bytes((void**)p, bytes);
}
template <class T>
cudaError_t device_alloc_async(T** p, size_t bytes, cudaStream_t s) {
  return device_alloc_async_bytes((void**)p, bytes, s);
}

}  // namespace gwmb

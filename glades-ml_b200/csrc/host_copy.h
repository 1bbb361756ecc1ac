// Copies between device memory and ordinary (pageable) host memory.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace glb {

// Both return when the host side of the copy is complete; to_device's device side is complete too.  The data on the device
// must be complete (its producers synchronised).  `device` is current on the calling thread.
cudaError_t copy_to_host(void* dst, const void* d_src, size_t bytes, int device);
cudaError_t copy_to_device(void* d_dst, const void* src, size_t bytes, int device);

// Takes the page faults of a result's fresh memory while the device is still at work on the result.
void host_prefault(void* p, size_t bytes);

// Handles alive on a device: the copy threads' staging memory and streams go with the last one.
void host_copy_retain(int device);
void host_copy_release(int device);

}  // namespace glb

// Copies between pageable host vectors and the device (host_copy.cpp).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace cpsgpu {

// cudaMemcpyAsync on stream of the current device, the host side any memory.
// copy_to_device returns once src has been read, copy_to_host once dst holds
// the data (as cudaMemcpyAsync does for pageable memory); pinned host memory
// keeps cudaMemcpyAsync's own ordering (asynchronous).
void copy_to_device(cudaStream_t stream, void *dst, const void *src, size_t bytes);
void copy_to_host(cudaStream_t stream, void *dst, const void *src, size_t bytes);

// Gives back the staging buffers and copy threads (cpsgpu_finalize); the next
// pageable copy makes them anew.
void host_copy_finalize();

}  // namespace cpsgpu

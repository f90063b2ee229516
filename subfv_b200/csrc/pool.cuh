// Stream-ordered device memory from a per-device pool that keeps freed memory (pool.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace subfv {

// *ptr: `bytes` of the current device's memory, usable on s from here on
int pool_alloc(void** ptr, size_t bytes, cudaStream_t s);
// gives it back after the work queued on s, or (idle) when no work uses it any more
void pool_free(void* ptr, cudaStream_t s);
void pool_free_idle(void* ptr);

}  // namespace subfv

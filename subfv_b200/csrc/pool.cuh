// Stream-ordered device memory from a per-device pool that keeps freed memory (pool.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace subfv {

// *p: `bytes` of device memory usable on s from here on; released with cudaFreeAsync
int pool_alloc(void** p, size_t bytes, cudaStream_t s);

}  // namespace subfv

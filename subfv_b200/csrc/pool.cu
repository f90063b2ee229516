// Device memory of states and batch slots, from one stream-ordered pool per device.
//
// A host code that calls the module procedures one at a time makes and drops a state per
// call, and a batch admits and retires problems all the time; cudaMalloc / cudaFree then
// cost more than the kernels (and cudaFree waits for the device), and the default pool
// gives its memory back to the system at every synchronisation. The pool here keeps up to
// kKept bytes of freed memory for the next state, gives back what exceeds it at
// synchronisations, and leaves the ordering between streams and threads to the runtime.
// A residual of 480 cells through compute_rhs_ns took 0.9 ms and more of which 0.1 ms on
// the device.
//
// The runtime's release threshold counts what the pool holds, memory in use included. So it
// follows the bytes in use, in steps of kStep: at a fixed threshold a program whose states
// pass it would keep nothing, and map and unmap memory with each state and each read-back
// through a staging buffer (1-3 ms a problem).
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "pool.cuh"

namespace subfv {

namespace {
constexpr int kMaxDevices = 64;
constexpr unsigned long long kKept = 512ull << 20, kStep = 64ull << 20;

struct Pool {
  cudaMemPool_t pool = nullptr;
  unsigned long long used = 0, threshold = 0;
};
struct Block {
  int dev;
  size_t bytes;
};
std::mutex g_pool_mutex;
Pool g_pool[kMaxDevices];
std::unordered_map<void*, Block> g_blocks;  // the allocations in use

// the bytes in use rounded up, and kKept more
void follow_use(Pool& p) {
  unsigned long long keep = (p.used + kStep - 1) / kStep * kStep + kKept;
  if (keep == p.threshold) return;
  p.threshold = keep;
  cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

int device_pool(int dev) {
  Pool& p = g_pool[dev];
  if (p.pool) return 0;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  SUBFV_CUDA(cudaMemPoolCreate(&p.pool, &props));
  return 0;
}

// the block leaves the books (before it is freed: afterwards its address may be another's)
void forget(void* ptr) {
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  auto it = g_blocks.find(ptr);
  if (it == g_blocks.end()) return;
  Pool& p = g_pool[it->second.dev];
  p.used -= it->second.bytes;
  g_blocks.erase(it);
  follow_use(p);
}
}  // namespace

int pool_alloc(void** ptr, size_t bytes, cudaStream_t s) {
  int dev = 0;
  SUBFV_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("pool_alloc: device index out of range");
    return -1;
  }
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (device_pool(dev)) return -1;
  Pool& p = g_pool[dev];
  SUBFV_CUDA(cudaMallocFromPoolAsync(ptr, bytes, p.pool, s));
  g_blocks[*ptr] = {dev, bytes};
  p.used += bytes;
  follow_use(p);
  return 0;
}

void pool_free(void* ptr, cudaStream_t s) {
  if (!ptr) return;
  forget(ptr);
  cudaFreeAsync(ptr, s);
}

void pool_free_idle(void* ptr) {
  if (!ptr) return;
  forget(ptr);
  cudaFree(ptr);
}

}  // namespace subfv

// The per-kernel entry points' scratch pool (scratch.h).
#include "../kernels/scratch.h"

#include <algorithm>
#include <cstdint>
#include <mutex>

namespace gpl {

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};

cudaError_t pool_of_device(cudaMemPool_t *pool) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess) return e;
    uint64_t keep = kScratchKeep;
    if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return e;
    }
    g_pool[dev] = p;
  }
  *pool = g_pool[dev];
  return cudaSuccess;
}
}  // namespace

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  cudaMemPool_t pool;
  cudaError_t e = pool_of_device(&pool);
  if (e != cudaSuccess) return e;
  return cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), pool, s);
}

}  // namespace gpl

// The per-kernel entry points' scratch pool (scratch.h).
#include "../kernels/scratch.h"

#include <cuda.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <type_traits>

namespace gpl {

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mutex;
// A device's pool, the primary context it was made under and the context of the last call. A
// device reset ends the pool with the primary context, whose successor has another number; the
// handle must not be used then (nor destroyed: the reset has).
struct DevicePool {
  cudaMemPool_t pool = nullptr;
  unsigned long long primary = 0, last = 0;
};
DevicePool g_pool[kMaxDevices];

// The driver's calls for contexts' numbers (NULL where the driver lacks one).
struct Driver {
  CUresult (*id)(CUcontext, unsigned long long *) = nullptr;
  CUresult (*state)(CUdevice, unsigned int *, int *) = nullptr;
  CUresult (*retain)(CUcontext *, CUdevice) = nullptr;
  CUresult (*release)(CUdevice) = nullptr;
  Driver() {
    auto look = [](const char *name, auto *fn) {
      void *p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) *fn = reinterpret_cast<std::remove_reference_t<decltype(*fn)>>(p);
    };
    look("cuCtxGetId", &id);
    look("cuDevicePrimaryCtxGetState", &state);
    look("cuDevicePrimaryCtxRetain", &retain);
    look("cuDevicePrimaryCtxRelease", &release);
    if (!id || !state || !retain || !release) id = nullptr;
  }
  unsigned long long current() const {
    unsigned long long n = 0;
    return id && id(nullptr, &n) == CUDA_SUCCESS ? n : 0;
  }
  // 0 while it is not active (a caller with contexts of its own)
  unsigned long long primary(int dev) const {
    unsigned int flags = 0;
    int active = 0;
    unsigned long long n = 0;
    CUcontext c = nullptr;
    if (!id || state(dev, &flags, &active) != CUDA_SUCCESS || !active || retain(&c, dev) != CUDA_SUCCESS) return 0;
    if (id(c, &n) != CUDA_SUCCESS) n = 0;
    release(dev);
    return n;
  }
};

cudaError_t pool_of_device(cudaMemPool_t *pool) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  static const Driver driver;
  std::lock_guard<std::mutex> lock(g_mutex);
  DevicePool &g = g_pool[dev];
  if (!g.pool || driver.current() != g.last) {
    if (!g.pool || driver.primary(dev) != g.primary) {
      g.pool = nullptr;
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
      g.pool = p;
      g.primary = driver.primary(dev);  // the first call on a device makes the context
    }
    g.last = driver.current();
  }
  *pool = g.pool;
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

// Device scratch of the per-kernel entry points, stream-ordered, from a pool of this library's
// own per device. The device's default pool gives freed memory back at every synchronisation
// (unless a context has raised its threshold), so a call that allocates and then synchronises
// maps new memory each time (0.1 to 0.4 ms for a few hundred KB); this pool keeps up to
// kScratchKeep bytes between calls and returns what is above that. Safe from any thread and
// stream, as the CUDA pool is.
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

namespace gpl {

constexpr size_t kScratchKeep = (size_t)64 << 20;
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s);
inline void scratch_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

// A scratch block for the scope of a call: freed, in stream order, when it goes.
class Scratch {
 public:
  Scratch(size_t bytes, cudaStream_t s) : s_(s), err_(scratch_alloc(&p_, bytes, s)) {}
  ~Scratch() { scratch_free(p_, s_); }
  Scratch(const Scratch &) = delete;
  Scratch &operator=(const Scratch &) = delete;
  cudaError_t error() const { return err_; }
  void *get() const { return p_; }

 private:
  void *p_ = nullptr;
  cudaStream_t s_;
  cudaError_t err_;
};

}  // namespace gpl

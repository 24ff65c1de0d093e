// Kernel attributes (the dynamic shared memory a launch may ask for) belong to
// a kernel on a device, and one process may hold contexts on several devices,
// in several threads.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace vfs {

// Runs f (which returns a cudaError_t) on the first call on each device;
// later calls return cudaSuccess at once.  A failure is returned and not
// remembered, so the next call tries again.  f may run twice when two threads
// meet: it sets attributes to constants.
struct PerDevice {
  std::atomic<unsigned long long> done{0};
  template <typename F>
  cudaError_t on(int device, F&& f) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = f();
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
  template <typename F>
  cudaError_t operator()(F&& f) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    return e != cudaSuccess ? e : on(device, f);
  }
};

// Lets a kernel take `bytes` of dynamic shared memory on the current device.
template <typename K>
inline cudaError_t allow_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace vfs

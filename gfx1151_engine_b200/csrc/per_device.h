// per_device.h -- what is set or looked up once for every GPU that a process uses. A kernel's attributes belong to
// one GPU's context: set for the first one alone, launches on a second GPU with more than 48 KB of shared memory fail. Host only.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace b200moe {

constexpr int kPerDeviceMax = 64;  // GPUs that are remembered; beyond, everything is done every time

class OncePerDevice {
 public:
  // set() if it has not succeeded on the current GPU yet. Threads that come at the same time may both do it, none goes on before it is done.
  template <typename F>
  cudaError_t operator()(F&& set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < kPerDeviceMax ? 1ull << dev : 0;
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = set();
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

// Multiprocessors of the current GPU.
inline cudaError_t sm_count(int* sms) {
  static std::atomic<int> known[kPerDeviceMax];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  *sms = dev < kPerDeviceMax ? known[dev].load(std::memory_order_relaxed) : 0;
  if (*sms > 0) return cudaSuccess;
  e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess && dev < kPerDeviceMax) known[dev].store(*sms, std::memory_order_relaxed);
  return e;
}

}  // namespace b200moe

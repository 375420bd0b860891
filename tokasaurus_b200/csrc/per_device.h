// Shared memory beyond 48 KB a block has to be asked for on every device that runs the kernel: one of these stands, static, beside
// the launch and remembers by device that it was.  (A flag for the whole process left the second device of a process without.)
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>
#include <initializer_list>

namespace tkb {

class SharedMemoryRequest {
 public:
  struct Kernel {
    const void* function;
    int bytes;
  };
  // 0, or the error of the call that failed (which is made again next time).
  int operator()(std::initializer_list<Kernel> kernels) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    const uint64_t bit = device < 64 ? 1ull << device : 0;  // (devices from 64 on are asked every time)
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    for (const Kernel& k : kernels) {
      e = cudaFuncSetAttribute(k.function, cudaFuncAttributeMaxDynamicSharedMemorySize, k.bytes);
      if (e != cudaSuccess) return (int)e;
    }
    done_.fetch_or(bit, std::memory_order_release);
    return 0;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace tkb

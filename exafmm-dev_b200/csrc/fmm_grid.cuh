// A barrier of all blocks of a launch whose blocks are resident together, for the kernels that
// run many small dependent steps: a cooperative launch (cudaLaunchCooperativeKernel), or a launch
// of one thread-block cluster.
#pragma once
#include <cuda_runtime.h>

namespace fmmb200 {

// The barrier of a cooperative launch counts arrivals up; a block that waits longer than
// kSyncSpins polls (seconds) sets *fault and every block leaves at its next barrier.  One
// cluster's is the hardware's (0.3 us instead of 1.5-2).
constexpr int kSyncSpins = 1 << 24;

struct GridBarrier {
  unsigned* arrived;  // zero before the launch
  int* fault;
  unsigned epoch;
  bool cluster;  // the launch is one cluster
  // all blocks' writes before it are visible to all blocks after it; false: leave the kernel
  __device__ __forceinline__ bool sync() {
    if (cluster) {
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
      return true;
    }
    __shared__ int ok;
    __syncthreads();
    epoch += gridDim.x;
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(arrived, 1u);
      int good = 1;
      for (int spin = 0;; spin++) {
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
        if (seen >= epoch) break;
        if (spin == kSyncSpins) {
          atomicExch(fault, 1);
          good = 0;
          break;
        }
      }
      __threadfence();
      if (good && *(volatile int*)fault) good = 0;
      ok = good;
    }
    __syncthreads();
    return ok != 0;
  }
};

}  // namespace fmmb200

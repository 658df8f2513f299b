// Host build of the C ABI's error path (exafmm-dev_b200/csrc/fmm_handle.cuh) over a fake of the
// CUDA runtime that counts the waits on each stream, for tests/test_error_path.py.
#include <cuda_runtime.h>

// device functions that the headers name and nothing here calls
struct Idx { unsigned x; };
static Idx threadIdx;
float __fadd_rn(float, float); double __dadd_rn(double, double);
float __fsub_rn(float, float); double __dsub_rn(double, double);
float __fmul_rn(float, float); double __dmul_rn(double, double);
float __fdiv_rn(float, float); double __ddiv_rn(double, double);
float __fsqrt_rn(float); double __dsqrt_rn(double);
float rsqrtf(float); double rsqrt(double);

#include "fmm_handle.cuh"

namespace fmmb200 {
std::atomic<long long> g_launches{0}, g_device_allocs{0};
}
using namespace fmmb200;

static int waits[4];  // by stream: the main one (1), the side streams (2, 3)
static cudaError_t wait_result = cudaSuccess;

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  waits[reinterpret_cast<size_t>(st) & 3]++;
  return wait_result;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) {
  *p = nullptr;
  return cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void*) { return cudaSuccess; }

// a call that ends as `how` says: 0 well, 1 an error of the library, 2 another exception, 3 no
// device memory left, 4 an error while the waits fail too; sides: the handle has its side
// streams.  n[0..2]: the waits on the streams; returns the status
int failed_call(int how, int sides, int* n) {
  Solver<float> s;
  fmm_b200_solver h;
  h.base = &s;
  s.cfg = fmm_b200_config{};
  s.stream = reinterpret_cast<cudaStream_t>(1);
  if (sides) {
    s.side = reinterpret_cast<cudaStream_t>(2);
    s.side_lo = reinterpret_cast<cudaStream_t>(3);
  }
  for (int& w : waits) w = 0;
  wait_result = how == 4 ? cudaErrorIllegalState : cudaSuccess;
  const int rc = guarded(&h, [&] {
    if (how == 1 || how == 4) throw FmmError(FMM_ERR_NOT_SUPPORTED, "no");
    if (how == 2) throw std::runtime_error("no");
    if (how == 3) s.keys.ensure(1000);
  });
  for (int k = 0; k < 3; k++) n[k] = waits[k + 1];
  return s.err.empty() == (how == 0) ? rc : -1;
}
}

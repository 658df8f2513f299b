// Utilities behind the C ABI: FP64 direct summation on the GPU (Traversal::direct +
// normalize, include/traversal.h:304-337, accumulated in double), the FP32 FMA throughput
// probe used as the roofline denominator of the FP32-pipe kernels, and the count of this
// library's kernel launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <mutex>
#include <string>

#include "fmm_solver.cuh"

namespace fmmb200 {
std::atomic<long long> g_launches{0};
std::atomic<long long> g_device_allocs{0};
}
using namespace fmmb200;

namespace {

// FP64 direct sum: a block takes 64 targets and one slice of the sources, its four groups of
// 64 threads every fourth source of each staged tile; the groups' sums meet in shared
// memory, the slices' in k_direct_sum, in slice order.  Bound by the FP64 pipe (about 22
// operations a pair with the reciprocal square root).  The slices fill the GPU whatever the
// number of targets: with a thread per target and no slices, 1,024 targets were four blocks
// (2^20 sources: 183 ms of kernel, now 2.0; the whole call takes 4.5 to 9 ms, the rest of it the
// allocation and the copies of pageable host memory, whose time varies that much).
constexpr int kDirTile = 256;
constexpr int kDirTargets = 64;
constexpr int kDirBlocks = 148 * 4;  // blocks wanted on the GPU: one wave at 4 per SM

// slices of the sources for nt targets: at most one wave of blocks, no slice shorter than a
// tile (so slices > 1 means at most kDirPartials partial sums)
constexpr size_t kDirPartials = 4 * (size_t)kDirTargets * kDirBlocks;
int direct_slices(int nt, int ns) {
  const int s = std::min(kDirBlocks / ceil_div(nt, kDirTargets), ceil_div(ns, kDirTile));
  return std::max(s, 1);
}

// the sums of slice blockIdx.y into out[4 (blockIdx.y nt + target)]
__global__ void __launch_bounds__(kDirTile, 4)
    k_direct(int nt, const double* __restrict__ xt, int ns, const double* __restrict__ xs,
             const double* __restrict__ qs, double eps2, int slice, double* __restrict__ out) {
  __shared__ double2 sh[kDirTile][2];
  const int i = blockIdx.x * kDirTargets + (threadIdx.x & (kDirTargets - 1));
  const int sub = threadIdx.x / kDirTargets;
  double x = 0, y = 0, z = 0;
  if (i < nt) {
    x = xt[3 * (size_t)i];
    y = xt[3 * (size_t)i + 1];
    z = xt[3 * (size_t)i + 2];
  }
  double pot = 0, ax = 0, ay = 0, az = 0;
  const long long first = (long long)blockIdx.y * slice;
  const int end = (int)(first + slice < ns ? first + slice : ns);
  for (long long j0 = first; j0 < end; j0 += kDirTile) {
    const size_t j = (size_t)j0 + threadIdx.x;
    __syncthreads();
    if (j < (size_t)end) {
      sh[threadIdx.x][0] = make_double2(xs[3 * j], xs[3 * j + 1]);
      sh[threadIdx.x][1] = make_double2(xs[3 * j + 2], qs[j]);
    }
    __syncthreads();
    const int cnt = (int)(end - j0 < kDirTile ? end - j0 : kDirTile);
#pragma unroll 4
    for (int k = sub; k < cnt; k += kDirTile / kDirTargets) {
      const double2 a = sh[k][0], b = sh[k][1];
      const double dx = a.x - x, dy = a.y - y, dz = b.x - z;
      const double r2 = dx * dx + dy * dy + dz * dz + eps2;
      if (r2 != 0) {
        const double inv = rsqrt(r2);
        const double qi = b.y * inv;
        const double inv3 = qi * inv * inv;
        pot += qi;
        ax += dx * inv3;
        ay += dy * inv3;
        az += dz * inv3;
      }
    }
  }
  __syncthreads();
  sh[threadIdx.x][0] = make_double2(pot, ax);
  sh[threadIdx.x][1] = make_double2(ay, az);
  __syncthreads();
  if (sub == 0 && i < nt) {
    for (int g = 1; g < kDirTile / kDirTargets; g++) {
      const double2 a = sh[threadIdx.x + g * kDirTargets][0],
                    b = sh[threadIdx.x + g * kDirTargets][1];
      pot += a.x;
      ax += a.y;
      ay += b.x;
      az += b.y;
    }
    double* o = out + 4 * ((size_t)blockIdx.y * nt + i);
    o[0] = pot;
    o[1] = ax;
    o[2] = ay;
    o[3] = az;
  }
}

__global__ void k_direct_sum(int n, int slices, const double* __restrict__ part,
                             double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double v = 0;
  for (int s = 0; s < slices; s++) v += part[(size_t)s * n + t];
  out[t] = v;
}

// device arrays in, 4 nt sums out; part: room for 4 nt `slices` doubles (slices > 1)
void launch_direct(int nt, const double* xt, int ns, const double* xs, const double* qs,
                   double eps2, int slices, double* part, double* out, cudaStream_t st) {
  const int len = ceil_div(ceil_div(ns, slices), kDirTile) * kDirTile;
  k_direct<<<dim3(ceil_div(nt, kDirTargets), slices), kDirTile, 0, st>>>(
      nt, xt, ns, xs, qs, eps2, len, slices > 1 ? part : out);
  FMM_LAUNCH_CHECK();
  if (slices > 1) {
    k_direct_sum<<<ceil_div(4LL * nt, 128), 128, 0, st>>>(4 * nt, slices, part, out);
    FMM_LAUNCH_CHECK();
  }
}

// independent FMA chains: 8 per thread, ITER iterations, 2 flops each
template <int ITER>
__global__ void __launch_bounds__(256) k_fma_probe(float* out, float s) {
  float a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) a[k] = threadIdx.x * 1e-7f + k;
#pragma unroll 16
  for (int i = 0; i < ITER; i++)
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = fmaf(a[k], s, 1e-7f);
  float t = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) t += a[k];
  if (t == 123.456f) out[0] = t;  // keeps the chains live
}

// ---- FP64 direct sum without allocation (fmm_b200_direct_noalloc) ---------------------
// The staging buffers of fmm_b200_direct (targets, sources, charges, output) live in one
// fixed array in device memory instead of per-call cudaMalloc/cudaFree.  Layout for a call
// (nt, ns), in doubles: targets [0, 3 nt), sources [3 nt, 3 nt + 3 ns), charges next (ns),
// output next (4 nt), the slices' partial sums next: at most 7 * 32768 + 4 * 65536 + 151,552
// = 643,072 doubles (4.91 MiB) per device.  No part of it has to start at zero: a call copies in
// every input it reads and the kernel writes every output that is copied back.
constexpr int kNoAllocMaxTargets = FMM_DIRECT_NOALLOC_MAX_TARGETS;
constexpr int kNoAllocMaxSources = FMM_DIRECT_NOALLOC_MAX_SOURCES;
constexpr size_t kNoAllocDoubles =
    7 * (size_t)kNoAllocMaxTargets + 4 * (size_t)kNoAllocMaxSources + kDirPartials;
static __device__ __align__(256) double g_direct_scratch[kNoAllocDoubles];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_base[kNoAllocMaxDevices] = {};
cudaStream_t g_noalloc_stream[kNoAllocMaxDevices] = {};

// Set-up of one device (which must be current), done once: the device address of the array
// (host code only sees a host-side stand-in under the array's name) and the call's own
// non-blocking stream (creating a stream allocates no device memory), so that the call
// neither waits for nor holds up the caller's other streams, the legacy default stream's
// implicit synchronisation included.
void noalloc_setup(int device, double** base, cudaStream_t* stream) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_base[device]) {
    void* p = nullptr;
    FMM_CUDA(cudaGetSymbolAddress(&p, g_direct_scratch));
    cudaStream_t st = nullptr;
    FMM_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    g_noalloc_stream[device] = st;
    g_noalloc_base[device] = static_cast<double*>(p);
  }
  *base = g_noalloc_base[device];
  *stream = g_noalloc_stream[device];
}

}  // namespace

extern "C" {

long long fmm_b200_kernel_launches(void) { return g_launches.load(); }
long long fmm_b200_device_allocations(void) { return g_device_allocs.load(); }

int fmm_b200_direct_noalloc(int device, int nt, const double* xt, int ns, const double* xs,
                            const double* qs, double eps2, double* out) {
  fmmb200::set_call_error("");
  if (nt < 0 || ns < 0 || (nt > 0 && (!xt || !out)) || (ns > 0 && (!xs || !qs)) ||
      device < 0 || device >= kNoAllocMaxDevices) {
    fmmb200::set_call_error("fmm_b200_direct_noalloc: invalid argument");
    return FMM_ERR_INVALID;
  }
  if (nt > kNoAllocMaxTargets || ns > kNoAllocMaxSources) {
    char msg[200];
    std::snprintf(msg, sizeof msg,
                  "fmm_b200_direct_noalloc: %d targets / %d sources exceed the static scratch "
                  "limits of %d targets / %d sources (fmm_b200_direct has none)",
                  nt, ns, kNoAllocMaxTargets, kNoAllocMaxSources);
    fmmb200::set_call_error(msg);
    return FMM_ERR_INVALID;
  }
  if (nt == 0) return FMM_OK;
  try {
    FMM_CUDA(cudaSetDevice(device));
    double* base = nullptr;
    cudaStream_t st = nullptr;
    noalloc_setup(device, &base, &st);
    double *dxt = base, *dxs = base + 3 * (size_t)nt, *dqs = dxs + 3 * (size_t)ns,
           *dout = dqs + ns;
    FMM_CUDA(cudaMemcpyAsync(dxt, xt, 24 * (size_t)nt, cudaMemcpyHostToDevice, st));
    if (ns) {
      FMM_CUDA(cudaMemcpyAsync(dxs, xs, 24 * (size_t)ns, cudaMemcpyHostToDevice, st));
      FMM_CUDA(cudaMemcpyAsync(dqs, qs, 8 * (size_t)ns, cudaMemcpyHostToDevice, st));
    }
    double* part = dout + 4 * (size_t)nt;
    launch_direct(nt, dxt, ns, dxs, dqs, eps2, direct_slices(nt, ns), part, dout, st);
    FMM_CUDA(cudaMemcpyAsync(out, dout, 32 * (size_t)nt, cudaMemcpyDeviceToHost, st));
    FMM_CUDA(cudaStreamSynchronize(st));
  } catch (const FmmError& e) {
    fmmb200::set_call_error(e.what());
    return e.code;
  }
  return FMM_OK;
}

int fmm_b200_direct(int device, int nt, const double* xt, int ns, const double* xs,
                    const double* qs, double eps2, double* out) {
  fmmb200::set_call_error("");
  if (nt < 0 || ns < 0 || (nt > 0 && (!xt || !out)) || (ns > 0 && (!xs || !qs))) {
    fmmb200::set_call_error("fmm_b200_direct: invalid argument");
    return FMM_ERR_INVALID;
  }
  if (nt == 0) return FMM_OK;
  try {
    FMM_CUDA(cudaSetDevice(device));
    DevArr<double> b;
    const int slices = direct_slices(nt, ns);
    b.ensure(3 * (size_t)nt + 4 * (size_t)ns + 4 * (size_t)nt * (slices > 1 ? 1 + slices : 1));
    double *dxt = b.p, *dxs = b.p + 3 * (size_t)nt, *dqs = dxs + 3 * (size_t)ns,
           *dout = dqs + ns;
    FMM_CUDA(cudaMemcpy(dxt, xt, 24 * (size_t)nt, cudaMemcpyHostToDevice));
    if (ns) {
      FMM_CUDA(cudaMemcpy(dxs, xs, 24 * (size_t)ns, cudaMemcpyHostToDevice));
      FMM_CUDA(cudaMemcpy(dqs, qs, 8 * (size_t)ns, cudaMemcpyHostToDevice));
    }
    launch_direct(nt, dxt, ns, dxs, dqs, eps2, slices, dout + 4 * (size_t)nt, dout, nullptr);
    FMM_CUDA(cudaMemcpy(out, dout, 32 * (size_t)nt, cudaMemcpyDeviceToHost));
    b.release();
  } catch (const FmmError& e) {
    fmmb200::set_call_error(e.what());
    return e.code;
  }
  return FMM_OK;
}

int fmm_b200_fp32_peak(int device, double* tflops) {
  if (!tflops) return FMM_ERR_INVALID;
  try {
    FMM_CUDA(cudaSetDevice(device));
    int sms = 0;
    FMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    DevArr<float> o;
    o.ensure(1);
    constexpr int ITER = 8192;
    const int blocks = sms * 8, threads = 256;
    k_fma_probe<ITER><<<blocks, threads>>>(o.p, 0.9999f);  // warm-up
    FMM_LAUNCH_CHECK();
    cudaEvent_t a, b;
    FMM_CUDA(cudaEventCreate(&a));
    FMM_CUDA(cudaEventCreate(&b));
    float best = 1e30f;
    for (int r = 0; r < 5; r++) {
      FMM_CUDA(cudaEventRecord(a));
      k_fma_probe<ITER><<<blocks, threads>>>(o.p, 0.9999f);
      FMM_LAUNCH_CHECK();
      FMM_CUDA(cudaEventRecord(b));
      FMM_CUDA(cudaEventSynchronize(b));
      float ms = 0;
      FMM_CUDA(cudaEventElapsedTime(&ms, a, b));
      best = ms < best ? ms : best;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    o.release();
    const double flops = 2.0 * 8 * ITER * (double)blocks * threads;
    *tflops = flops / (best * 1e-3) / 1e12;
  } catch (const FmmError& e) {
    return e.code;
  }
  return FMM_OK;
}

}  // extern "C"

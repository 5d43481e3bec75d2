// FP64 direct sum for sampled targets that allocates no memory.
//
// Why it exists: tapas_b200_direct keeps the partial sums (and a host call's
// targets and results) in device buffers of its context, which a larger call
// allocates anew.  Some callers cannot allow a
// device allocation where they check accuracy: a time-stepping loop that
// reserves all of its device memory up front (a cudaMalloc there can fail or
// push the solver out of memory), or code that shares the GPU with other
// streams (cudaMalloc / cudaFree synchronise the whole device and stall that
// work).  This entry point takes only caller-owned device buffers and keeps
// its partial sums in one fixed device array compiled into the library.
//
// Limits and sharing:
//  - at most kMaxTargets targets per call; more are rejected with
//    TAPAS_B200_ERR_CAPACITY and a message;
//  - the scratch array (kMaxRows x 4 doubles = 2 MiB) exists once
//    per GPU that loads the library and is held until the process exits;
//  - every call on a device uses the same array, and it keeps the last call's
//    contents.  Each call writes every slot it later reads, so nothing needs
//    clearing; calls that overlap on the GPU (different streams, or different
//    host threads without ordering) race on the array and must be serialised
//    by the caller;
//  - the first call on a device looks up the array's device address
//    (cudaGetSymbolAddress, with that device current) and caches it; make
//    that first call before any stream capture.
#include <mutex>

#include "common.cuh"
#include "direct.cuh"

namespace tb {
namespace {

constexpr int kMaxTargets = 4096;
constexpr int64_t kMaxRows = 65536;  // (target, split) pairs: 16 splits of the most targets
constexpr int kMaxDevices = 64;

// The scratch: per (target, split) the 4 partial sums.
static __device__ __align__(256) double g_direct_scratch[(size_t)kMaxRows * 4];

double *g_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mutex;

}  // namespace
}  // namespace tb

using namespace tb;

extern "C" int tapas_b200_direct_noalloc(const double *x, const double *y, const double *z,
                                         const double *q, int64_t n, const int64_t *targets,
                                         int64_t k, double *out4, void *stream) {
  if (!x || !y || !z || !q || !targets || !out4 || n <= 0 || k <= 0) {
    set_error(nullptr, "direct_noalloc: need n > 0, k > 0 and non-null device pointers");
    return TAPAS_B200_ERR_ARG;
  }
  if (k > kMaxTargets) {
    set_error(nullptr,
              "direct_noalloc: %lld targets exceed the fixed scratch capacity of %d targets "
              "per call; split the target list",
              (long long)k, kMaxTargets);
    return TAPAS_B200_ERR_CAPACITY;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    set_error(nullptr, "direct_noalloc: no usable current device (%s)", cudaGetErrorString(e));
    return TAPAS_B200_ERR_CUDA;
  }
  double *scratch;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
      // Host code cannot use g_direct_scratch's name as a device address:
      // look the address up once for this device (the current one).
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, g_direct_scratch);
      if (e != cudaSuccess || !p) {
        set_error(nullptr, "direct_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                  cudaGetErrorString(e));
        return TAPAS_B200_ERR_CUDA;
      }
      g_scratch_addr[dev] = static_cast<double *>(p);
    }
    scratch = g_scratch_addr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // An error left by earlier asynchronous work would otherwise be read back
  // after the launch below and reported as this call's launch failure.
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(nullptr, "direct_noalloc: a CUDA error from earlier work was pending: %s",
              cudaGetErrorString(e));
    return TAPAS_B200_ERR_CUDA;
  }
  int num_sms = 0;
  e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) {
    set_error(nullptr, "direct_noalloc: %s", cudaGetErrorString(e));
    return TAPAS_B200_ERR_CUDA;
  }
  // the scratch has room for 16 splits of any k: 4096 targets x 1M bodies 5.04 ms, 5.14 with
  // the rule's 7, whose last wave of blocks is nearly empty
  const int64_t most = std::max<int64_t>(1, n / (16 * kDirectThreads));
  const int nsplit = (int)std::min<int64_t>(
      kMaxRows / k, std::max<int64_t>(direct_splits(num_sms, n, k),
                                      std::min<int64_t>(kMaxRows / kMaxTargets, most)));
  direct_tiles<<<dim3((unsigned)((k + kDirectTargets - 1) / kDirectTargets), nsplit),
                 kDirectThreads, 0, s>>>(x, y, z, q, n, targets, k, nsplit, scratch);
  e = cudaGetLastError();
  if (e == cudaSuccess) {
    direct_finish<<<(unsigned)((k * 4 + 255) / 256), 256, 0, s>>>(scratch, k, nsplit, out4);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    set_error(nullptr, "direct_noalloc: launch failed: %s", cudaGetErrorString(e));
    return TAPAS_B200_ERR_CUDA;
  }
  return TAPAS_B200_OK;
}

// scratch.cpp -- stream-ordered scratch memory of the library's launches.
//
// Scratch comes from one memory pool per device that keeps up to kKeepBytes
// between launches.  The device's default pool gives freed memory back to
// the driver at every synchronization, so each launch after one mapped its
// scratch anew: 40-100 us of host time per gbv_render (GB300, 256 bytes of
// scratch).  The pool orders reuse by the streams' own work, is safe to use
// from several threads and streams, and does not make one stream wait for
// another to reuse its memory.  The largest request is a frame's fragment log
// (512 MB); release_scratch gives back what no launch holds.
#include <mutex>
#include <cuda_runtime.h>
#include "gbv_internal.h"

namespace gbv {
namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKeepBytes = 576ull << 20;
std::mutex g_mutex;
cudaMemPool_t g_pools[kMaxDevices];

// The pool of device `dev` (made on first use); null if it cannot be made.
// `stale`: a pool whose handle is no longer valid (a device reset destroys
// pools behind their handles), to be made anew.
cudaMemPool_t device_pool(int dev, cudaMemPool_t stale) {
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_pools[dev] && g_pools[dev] != stale) return g_pools[dev];
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    pool = nullptr;
  } else {
    unsigned long long keep = kKeepBytes;
    int off = 0;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &off);
  }
  g_pools[dev] = pool;
  return pool;
}

}  // namespace

cudaError_t scratch_alloc(void **ptr, size_t bytes, cudaStream_t stream) {
  *ptr = nullptr;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  int dev = 0;
  cudaError_t e = cudaStreamIsCapturing(stream, &cap);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  // a captured allocation belongs to the graph, whatever pool it names
  cudaMemPool_t pool = cap == cudaStreamCaptureStatusNone ? device_pool(dev, nullptr) : nullptr;
  for (int attempt = 0; pool && attempt < 2; attempt++) {
    e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
    if (e != cudaErrorInvalidValue && e != cudaErrorInvalidResourceHandle) return e;  // the handle is valid
    cudaGetLastError();
    pool = device_pool(dev, pool);
  }
  return cudaMallocAsync(ptr, bytes, stream);
}

cudaError_t release_scratch(int dev) {
  cudaMemPool_t pool = nullptr;
  if (dev >= 0 && dev < kMaxDevices) {
    std::lock_guard<std::mutex> lock(g_mutex);
    pool = g_pools[dev];
  }
  return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

namespace {
// This thread's calls may allocate although another stream is being captured
// (which they do not touch), whatever that capture's mode.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
}  // namespace

bool optional_scratch(void **ptr, size_t bytes, cudaStream_t stream) {
  const RelaxedCapture relaxed;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  *ptr = nullptr;
  cudaError_t e = cudaStreamIsCapturing(stream, &cap);
  if (e == cudaSuccess && cap != cudaStreamCaptureStatusNone) return false;
  if (e == cudaSuccess) e = scratch_alloc(ptr, bytes, stream);
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  *ptr = nullptr;
  return false;
}

cudaError_t free_optional_scratch(void *ptr, cudaStream_t stream) {
  const RelaxedCapture relaxed;
  return ptr ? cudaFreeAsync(ptr, stream) : cudaSuccess;
}

}  // namespace gbv

/* The scratch pool against a fake CUDA runtime: which errors replace the
   pool, what a capture does, and that the memory kept is given back. */
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "cuda_runtime.h"

static int g_created, g_trimmed, g_allocated, g_default, g_freed;
static cudaError_t g_error;  // of the next allocations from a pool
static cudaStreamCaptureStatus g_capture;
static cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;
static cudaMemPool_t g_last;

cudaError_t cudaGetDevice(int *dev) { return *dev = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { return *s = g_capture, cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *mode) {
  const cudaStreamCaptureMode was = g_mode;
  g_mode = *mode;
  *mode = was;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) {
  *pool = (cudaMemPool_t)(size_t)(0x100 * ++g_created);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
  if (pool != g_last || keep != 0) return cudaErrorInvalidValue;
  g_trimmed++;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **ptr, size_t, cudaMemPool_t pool, cudaStream_t) {
  // an invalid handle: the pools made before the error was planted
  if (g_error == cudaErrorInvalidValue && pool != g_last) g_error = cudaSuccess;
  if (g_error != cudaSuccess) return g_error;
  g_last = pool;
  g_allocated++;
  *ptr = (void *)pool;
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **ptr, size_t, cudaStream_t) {
  g_default++;
  *ptr = (void *)0x1;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *, cudaStream_t) { return g_freed++, cudaSuccess; }

#include "../../barney_gb300/csrc/scratch.cpp"

#define CHECK(x)                                                    \
  do {                                                              \
    if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1; \
  } while (0)

int main() {
  using namespace gbv;
  void *p = nullptr;
  CHECK(release_scratch(0) == cudaSuccess && g_trimmed == 0);  // no pool yet
  CHECK(scratch_alloc(&p, 256, nullptr) == cudaSuccess && g_created == 1 && g_allocated == 1);
  // errors that leave the pool valid: returned, the pool is kept
  for (cudaError_t e : {cudaErrorMemoryAllocation, cudaErrorStreamCaptureUnsupported, cudaErrorIllegalAddress}) {
    g_error = e;
    CHECK(scratch_alloc(&p, 256, nullptr) == e);
    CHECK(g_created == 1 && g_default == 0);
    CHECK(!optional_scratch(&p, 256, nullptr) && p == nullptr);
    g_error = cudaSuccess;
  }
  CHECK(scratch_alloc(&p, 256, nullptr) == cudaSuccess && g_created == 1 && g_allocated == 2);
  // a handle that is no longer valid: a new pool
  g_error = cudaErrorInvalidValue;
  CHECK(scratch_alloc(&p, 256, nullptr) == cudaSuccess && g_created == 2 && g_allocated == 3);
  CHECK(release_scratch(0) == cudaSuccess && g_trimmed == 1);
  CHECK(release_scratch(-1) == cudaSuccess && release_scratch(1 << 20) == cudaSuccess && g_trimmed == 1);
  // a capture: a launch's own scratch belongs to the graph, what it can do without is not taken
  g_capture = cudaStreamCaptureStatusActive;
  CHECK(scratch_alloc(&p, 256, nullptr) == cudaSuccess && g_default == 1 && g_allocated == 3);
  CHECK(!optional_scratch(&p, 256, nullptr) && p == nullptr && g_default == 1);
  g_capture = cudaStreamCaptureStatusNone;
  CHECK(optional_scratch(&p, 256, nullptr) && p != nullptr && g_allocated == 4);
  CHECK(free_optional_scratch(p, nullptr) == cudaSuccess && g_freed == 1);
  CHECK(free_optional_scratch(nullptr, nullptr) == cudaSuccess && g_freed == 1);
  CHECK(g_mode == cudaStreamCaptureModeGlobal);  // as it was
  std::puts("ok");
  return 0;
}

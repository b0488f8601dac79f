/* The few declarations of the CUDA runtime that the library's scratch pool
   uses, for a build against a fake runtime (scratch_check.cpp). */
#pragma once
#include <stddef.h>

enum cudaError_t {
  cudaSuccess = 0,
  cudaErrorInvalidValue = 1,
  cudaErrorMemoryAllocation = 2,
  cudaErrorInvalidResourceHandle = 400,
  cudaErrorIllegalAddress = 700,
  cudaErrorStreamCaptureUnsupported = 900
};
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal = 0, cudaStreamCaptureModeRelaxed = 2 };
enum { cudaMemAllocationTypePinned = 1, cudaMemLocationTypeDevice = 1 };
enum cudaMemPoolAttr { cudaMemPoolReuseAllowInternalDependencies = 3, cudaMemPoolAttrReleaseThreshold = 4 };
typedef struct CUstream_st *cudaStream_t;
typedef struct CUmemPool_st *cudaMemPool_t;
struct float2 { float x, y; };
struct cudaMemPoolProps {
  int allocType, handleTypes;
  struct { int type, id; } location;
};

cudaError_t cudaGetDevice(int *dev);
cudaError_t cudaGetLastError();
cudaError_t cudaStreamIsCapturing(cudaStream_t stream, cudaStreamCaptureStatus *status);
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *mode);
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *props);
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t pool, cudaMemPoolAttr attr, void *value);
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep);
cudaError_t cudaMallocFromPoolAsync(void **ptr, size_t bytes, cudaMemPool_t pool, cudaStream_t stream);
cudaError_t cudaMallocAsync(void **ptr, size_t bytes, cudaStream_t stream);
cudaError_t cudaFreeAsync(void *ptr, cudaStream_t stream);

// A stand-in for the CUDA runtime, for tests of host code: "device" memory is host memory,
// streams do nothing, and an allocation or a synchronisation fails when a test says so.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

static size_t g_malloc_limit = ~(size_t)0;
static cudaError_t g_sync_result = cudaSuccess;
static int g_syncs = 0;
extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)8, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return ++g_syncs, g_sync_result; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)8, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)8, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (n > g_malloc_limit) return cudaErrorMemoryAllocation;
  return *p = std::calloc(n, 1), cudaSuccess;
}
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(n, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "stand-in"; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes*, const void*) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 1, cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}


struct psift_ctx;
namespace psift {
void jpeg_release(psift_ctx*) {}
void png_release(psift_ctx*) {}
}  // namespace psift

#define CHECK(x)                                                 \
  do {                                                           \
    if (!(x)) {                                                  \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #x); \
      return 1;                                                  \
    }                                                            \
  } while (0)

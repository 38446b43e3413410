// The few CUDA runtime calls of the library's host classes, on a machine without a device: two pretended devices, a count
// and a record of each call.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <vector>

namespace fake {
inline thread_local int device = 0;
inline std::atomic<int> streams{0}, mallocs{0}, frees{0};
inline std::atomic<int> stream_device{-1}, synced_device{-1};
__attribute__((weak)) cudaError_t sync_result = cudaSuccess;
}  // namespace fake

extern "C" {
__attribute__((weak)) cudaError_t cudaGetDevice(int* d) { return *d = fake::device, cudaSuccess; }
__attribute__((weak)) cudaError_t cudaSetDevice(int d) { return fake::device = d, cudaSuccess; }
__attribute__((weak)) cudaError_t cudaGetLastError() { return cudaSuccess; }
__attribute__((weak)) cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  for (volatile int i = 0; i < 200000; ++i) {  // as slow as the real one, so that callers meet in it
  }
  fake::stream_device = fake::device;
  *s = reinterpret_cast<cudaStream_t>(static_cast<size_t>(16 * ++fake::streams));
  return cudaSuccess;
}
__attribute__((weak)) cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
__attribute__((weak)) cudaError_t cudaDeviceSynchronize() { return fake::synced_device = fake::device, fake::sync_result; }
__attribute__((weak)) cudaError_t cudaMalloc(void** p, size_t) { return *p = std::malloc(16), ++fake::mallocs, cudaSuccess; }
__attribute__((weak)) cudaError_t cudaFree(void* p) { return std::free(p), ++fake::frees, cudaSuccess; }
}

#define CHECK(c)                                                       \
  do {                                                                 \
    if (!(c)) {                                                        \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c);     \
      std::exit(1);                                                    \
    }                                                                  \
  } while (0)

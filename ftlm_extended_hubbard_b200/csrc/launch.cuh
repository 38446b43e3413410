// Launches: the shared memory a kernel may use, and kernels without the gap of a launch between them.
//
// Kernels that follow one another on a stream without the gap of a launch (programmatic dependent launch).  A kernel
// that starts with x = follow<true>(x) may be launched with early = true: its blocks are then placed while the kernel
// before it drains, and wait in follow() until that kernel has ended and its writes are visible, so the order of all
// reads and writes is that of an ordinary launch.  Every thread of every block passes follow(), so the kernel's end
// implies that of all before it. Only where the vectors stay in L2 (kEarlyStates): there the gap is a large part of a
// kernel (two-pass H v, a call: 4x3 (5,6) 55.3 -> 51.6 us, 4x3 (4,4) 21.4 -> 17.2), while waiting blocks cost
// large sectors 1 to 2 % (5x3 (5,5) 506 -> 514 us).  Under stream capture the launches are ordinary ones.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ftlm_b200 {

// Allows a kernel `bytes` of dynamic shared memory, beside `own` of its static.  The limit is a property of the kernel that
// all threads share, so it is always set to the same value, the most there is: a call that set it to its own size could
// lower it between another thread's call and launch.
constexpr size_t kBlockShared = 227 * 1024;
template <class K>
cudaError_t allow_shared(K kernel, size_t bytes, size_t own = 0) {
  if (bytes + own > kBlockShared) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBlockShared - own));
}

constexpr int64_t kEarlyStates = int64_t(1) << 21;  // 16-byte elements of a vector: 32 MB

// Returns p, as a value that the wait makes: no load through it can move ahead of the wait, whatever the compiler knows
// of the pointer it came from.  Without kEarly just p: the loads of large sectors lose 1 to 3 % with the detour.
template <bool kEarly, class T>
__device__ __forceinline__ const T* follow(const T* p) {
  if constexpr (kEarly) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" : "+l"(p)::"memory");
  }
  return p;
}

inline bool early_ok(int64_t states, cudaStream_t st) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return states <= kEarlyStates && cudaStreamIsCapturing(st, &c) == cudaSuccess && c == cudaStreamCaptureStatusNone;
}

template <class... P, class... A>
cudaError_t launch_after(bool early, void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

}  // namespace ftlm_b200

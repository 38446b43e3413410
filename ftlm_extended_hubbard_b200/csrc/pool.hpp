// Device blocks kept between calls, for workspaces and tables that live for one call or one small sector: cudaMalloc and
// cudaFree cost tens of microseconds to milliseconds each, more than many of the calls.  Per device, at most kPoolKeep
// bytes stay here (given back by ftlm_gpu_batched_release, or when device memory runs out); thread-safe.  A block is
// given only when no work on it is in flight: the next owner may be on any stream.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

#include "lazy_stream.hpp"

namespace ftlm_b200 {
namespace capi {

constexpr size_t kPoolKeep = size_t(1) << 30;
cudaError_t pool_take(size_t bytes, void** p, size_t* got);
// idle = false: work on the block may be in flight, so it is freed (which waits) instead of kept.
void pool_give(void* p, size_t got, bool idle = true);
void pool_trim();

// Waits for a device's work, whatever device is current; whether it could (a stream capture forbids it).
inline bool device_idle(int device) {
  DeviceGuard on(device);
  return cudaDeviceSynchronize() == cudaSuccess;
}

// One array in a block of the pool; its owner gives it back when no work on it is in flight.
struct PoolBuf {
  void* p = nullptr;
  size_t got = 0;
  PoolBuf() = default;
  PoolBuf(const PoolBuf&) = delete;
  PoolBuf& operator=(const PoolBuf&) = delete;
  ~PoolBuf() { free(); }
  void free(bool idle = true) {
    if (p) pool_give(p, got, idle);
    p = nullptr;
    got = 0;
  }
  cudaError_t alloc(size_t bytes) {
    free();
    return pool_take(bytes, &p, &got);
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// One block of the pool, laid out by add() and obtained by commit().  idle() says that the work on it has ended; without
// it (an error on the way) the block is given back after the device has.
class Scratch {
 public:
  Scratch() = default;
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  ~Scratch() {
    if (p_) pool_give(p_, got_, !busy_ || device_idle(-1));
  }
  size_t add(size_t bytes) {
    const size_t at = size_;
    size_ += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
    return at;
  }
  template <class T>
  size_t array(size_t n) {
    return add(n * sizeof(T));
  }
  cudaError_t commit() { return pool_take(size_, &p_, &got_); }
  template <class T>
  T* at(size_t off) const {
    return reinterpret_cast<T*>(static_cast<char*>(p_) + off);
  }
  void idle() { busy_ = false; }
  void busy() { busy_ = true; }

 private:
  void* p_ = nullptr;
  size_t size_ = 0, got_ = 0;
  bool busy_ = true;
};

}  // namespace capi
}  // namespace ftlm_b200

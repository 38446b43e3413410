// A handle's own stream, and calls on its device whatever device is current.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace ftlm_b200 {
namespace capi {

// Makes a device current for a scope.
class DeviceGuard {
 public:
  explicit DeviceGuard(int device) {
    if (device < 0 || cudaGetDevice(&before_) != cudaSuccess || before_ == device) return;
    moved_ = cudaSetDevice(device) == cudaSuccess;
  }
  DeviceGuard(const DeviceGuard&) = delete;
  DeviceGuard& operator=(const DeviceGuard&) = delete;
  ~DeviceGuard() {
    if (moved_) cudaSetDevice(before_);
  }

 private:
  int before_ = 0;
  bool moved_ = false;
};

// A non-blocking stream, created when it is first asked for: a sweep's sectors mostly share one launch and need none.
// Several threads may ask at once. The stream is of the handle's device: launches on it with another device current are
// refused by the runtime, as they would be on a stream made with the handle.
class LazyStream {
 public:
  LazyStream() = default;
  LazyStream(const LazyStream&) = delete;
  LazyStream& operator=(const LazyStream&) = delete;
  ~LazyStream() {
    const cudaStream_t s = s_.load();
    if (s) cudaStreamDestroy(s);
  }
  void set_device(int device) { device_ = device; }
  operator cudaStream_t() {  // the legacy default stream where none can be created
    cudaStream_t s = s_.load(std::memory_order_acquire);
    if (s) return s;
    std::lock_guard<std::mutex> lock(mu_);
    s = s_.load(std::memory_order_acquire);
    if (s) return s;
    DeviceGuard on(device_);
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    s_.store(s, std::memory_order_release);
    return s;
  }

 private:
  std::mutex mu_;
  std::atomic<cudaStream_t> s_{nullptr};
  int device_ = -1;  // the current one
};

}  // namespace capi
}  // namespace ftlm_b200

// The kept device blocks (contract in pool.hpp).
#include "pool.hpp"

#include <map>
#include <mutex>
#include <new>
#include <vector>

namespace {

struct PoolBlock {
  void* p;
  size_t bytes;
};
struct DevicePool {
  std::vector<PoolBlock> free;
  size_t kept = 0;
};
struct Pool {
  std::mutex mu;
  std::map<int, DevicePool> devices;
  std::map<void*, int> device;  // of every block taken or kept
};
Pool& pool() {
  static Pool* p = new Pool;  // not destroyed: its blocks end with the context
  return *p;
}

}  // namespace

cudaError_t ftlm_b200::capi::pool_take(size_t bytes, void** p, size_t* got) {
  *p = nullptr;
  *got = 0;
  bytes = std::max<size_t>(bytes, 256);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Pool& P = pool();
  {
    std::lock_guard<std::mutex> lock(P.mu);
    DevicePool& D = P.devices[dev];
    auto& v = D.free;
    size_t best = v.size();
    for (size_t i = 0; i < v.size(); ++i)  // the smallest that fits, unless most of it would lie idle
      if (v[i].bytes >= bytes && v[i].bytes <= 8 * bytes + (size_t(1) << 20) && (best == v.size() || v[i].bytes < v[best].bytes))
        best = i;
    if (best < v.size()) {
      *p = v[best].p;
      *got = v[best].bytes;
      D.kept -= v[best].bytes;
      v[best] = v.back();
      v.pop_back();
      return cudaSuccess;
    }
  }
  size_t want = bytes;  // rounded up to an eighth of its power of two, so that blocks fit each other's uses
  size_t unit = 256;
  while (unit * 16 < bytes) unit *= 2;
  want = (bytes + unit - 1) / unit * unit;
  e = cudaMalloc(p, want);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    pool_trim();
    e = cudaMalloc(p, want);
  }
  if (e != cudaSuccess) return e;
  try {
    std::lock_guard<std::mutex> lock(P.mu);
    P.device[*p] = dev;
  } catch (const std::bad_alloc&) {
    cudaFree(*p);
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  *got = want;
  return cudaSuccess;
}

void ftlm_b200::capi::pool_give(void* p, size_t got, bool idle) {
  if (!p) return;
  Pool& P = pool();
  {
    std::lock_guard<std::mutex> lock(P.mu);
    auto it = P.device.find(p);
    if (it != P.device.end()) {
      DevicePool& D = P.devices[it->second];
      if (idle && D.kept + got <= kPoolKeep) {
        try {
          D.free.push_back(PoolBlock{p, got});
          D.kept += got;
          return;
        } catch (const std::bad_alloc&) {  // no room to note it
        }
      }
      P.device.erase(it);
    }
  }
  cudaFree(p);
}

void ftlm_b200::capi::pool_trim() {
  Pool& P = pool();
  std::vector<PoolBlock> all;
  {
    std::lock_guard<std::mutex> lock(P.mu);
    for (auto& d : P.devices) {
      all.insert(all.end(), d.second.free.begin(), d.second.free.end());
      d.second.free.clear();
      d.second.kept = 0;
    }
    for (const PoolBlock& b : all) P.device.erase(b.p);
  }
  for (const PoolBlock& b : all) cudaFree(b.p);
}

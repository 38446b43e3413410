// The kept device blocks with two devices, a capture in progress and more than they may hold.
#include "fake_runtime.hpp"
#include "pool.hpp"

using namespace ftlm_b200::capi;

int main() {
  void *a = nullptr, *b = nullptr;
  size_t ga = 0, gb = 0;
  // a handle of device 1 goes while device 0 is current: its own device is waited for, its block serves that device only
  fake::device = 1;
  CHECK(pool_take(5000, &a, &ga) == cudaSuccess && ga >= 5000);
  fake::device = 0;
  CHECK(device_idle(1));
  CHECK(fake::synced_device == 1 && fake::device == 0);
  pool_give(a, ga, true);
  CHECK(pool_take(5000, &b, &gb) == cudaSuccess && b != a);
  fake::device = 1;
  void* c = nullptr;
  size_t gc = 0;
  CHECK(pool_take(5000, &c, &gc) == cudaSuccess && c == a);
  // a device that cannot be waited for (a capture): the block is not handed to another owner
  fake::sync_result = cudaErrorStreamCaptureUnsupported;
  const int frees = fake::frees;
  pool_give(c, gc, device_idle(1));
  CHECK(fake::frees == frees + 1);
  int mallocs = fake::mallocs;
  CHECK(pool_take(5000, &c, &gc) == cudaSuccess && fake::mallocs == mallocs + 1);
  {
    Scratch s;
    s.add(5000);
    CHECK(s.commit() == cudaSuccess);
  }
  CHECK(fake::frees == frees + 2);
  fake::sync_result = cudaSuccess;
  // each device keeps its own gigabyte
  const size_t big = size_t(900) << 20;
  fake::device = 0;
  CHECK(pool_take(big, &a, &ga) == cudaSuccess);
  fake::device = 1;
  CHECK(pool_take(big, &b, &gb) == cudaSuccess);
  void* d = nullptr;
  size_t gd = 0;
  CHECK(pool_take(big, &d, &gd) == cudaSuccess);
  pool_give(a, ga);
  pool_give(b, gb);
  pool_give(d, gd);  // more than device 1 may keep
  CHECK(fake::frees == frees + 3);
  mallocs = fake::mallocs;
  CHECK(pool_take(big, &b, &gb) == cudaSuccess);
  fake::device = 0;
  CHECK(pool_take(big, &a, &ga) == cudaSuccess);
  CHECK(fake::mallocs == mallocs);
  return 0;
}

// Many threads ask a fresh handle for its stream at once, with another device current than the handle's.
#include "fake_runtime.hpp"
#include "lazy_stream.hpp"

#include <thread>

int main() {
  for (int round = 0; round < 50; ++round) {
    fake::streams = 0;
    ftlm_b200::capi::LazyStream s;
    s.set_device(1);
    std::vector<std::thread> pool;
    std::vector<cudaStream_t> got(8, nullptr);
    std::atomic<int> ready{0};
    for (int t = 0; t < 8; ++t)
      pool.emplace_back([&, t]() {
        ++ready;
        while (ready < 8) {
        }
        got[t] = s;
        CHECK(fake::device == 0);
      });
    for (auto& t : pool) t.join();
    CHECK(fake::streams == 1);
    CHECK(fake::stream_device == 1);
    for (auto g : got) CHECK(g == got[0] && g != nullptr);
  }
  return 0;
}

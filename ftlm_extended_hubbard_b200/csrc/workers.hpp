// Independent host work shared out among threads.
#pragma once

#include <atomic>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace ftlm_b200 {

// work(i) for 0 <= i < n, by the calling thread and up to threads - 1 others, which take the next i each.  Where no
// further thread can be started those there are do all of it; the first exception of any of them is thrown here, after
// all have ended.
template <class Work>
void share_out(int threads, int64_t n, Work&& work) {
  std::atomic<int64_t> next{0};
  std::exception_ptr error;
  std::mutex mu;
  auto run = [&]() {
    try {
      for (int64_t i; (i = next.fetch_add(1)) < n;) work(i);
    } catch (...) {
      next.store(n);
      std::lock_guard<std::mutex> lock(mu);
      if (!error) error = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  try {
    for (int t = 1; t < threads && t < n; ++t) pool.emplace_back(run);
  } catch (const std::exception&) {  // no more threads, or no memory to note one
  }
  run();
  for (auto& t : pool) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace ftlm_b200

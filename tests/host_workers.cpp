// Work shared out among threads: every item once, also with fewer threads than asked for, and an exception of any thread
// arrives in the caller.
#include "workers.hpp"

#include <cstdio>
#include <cstdlib>
#include <new>

#define CHECK(c)                                                       \
  do {                                                                 \
    if (!(c)) {                                                        \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c);     \
      std::exit(1);                                                    \
    }                                                                  \
  } while (0)

int main() {
  for (int threads : {0, 1, 2, 7, 64})
    for (int64_t n : {0, 1, 5, 1000}) {
      std::vector<std::atomic<int>> seen(static_cast<size_t>(n));
      ftlm_b200::share_out(threads, n, [&](int64_t i) { ++seen[static_cast<size_t>(i)]; });
      for (auto& s : seen) CHECK(s == 1);
    }
  const auto self = std::this_thread::get_id();
  for (bool in_caller : {false, true})
    for (int round = 0; round < 20; ++round) {
      bool caught = false;
      std::atomic<bool> thrown{false};
      try {
        ftlm_b200::share_out(8, 1 << 20, [&](int64_t) {
          if ((std::this_thread::get_id() == self) == in_caller && !thrown.exchange(true)) throw std::bad_alloc();
          while (!thrown) std::this_thread::yield();  // until the thread that is to throw has had an item
        });
      } catch (const std::bad_alloc&) {
        caught = true;
      }
      CHECK(caught);
    }
  return 0;
}

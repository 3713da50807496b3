// Host loops on several threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <exception>
#include <thread>
#include <vector>

namespace ptyb::eng {

// Runs fn(begin, end) over [0, n) on up to `most` host threads, each of at least `each` values.
// What no thread can be started for (a process limit, no memory) runs on the caller's; every
// started thread has ended when the function is left.
template <class F>
void parallel_range(size_t n, size_t each, size_t most, F&& fn) {
  const size_t nt = std::min<size_t>({most, std::max(1u, std::thread::hardware_concurrency()),
                                      n / each});
  size_t begin = 0;
  struct Joined {
    std::vector<std::thread> ts;
    ~Joined() {
      for (auto& t : ts) t.join();
    }
  } started;
  if (nt > 1) {
    const size_t chunk = (n + nt - 1) / nt;
    try {
      started.ts.reserve(nt);
      while (begin < n) {
        const size_t end = std::min(n, begin + chunk);
        started.ts.emplace_back([&fn, begin, end] { fn(begin, end); });
        begin = end;
      }
    } catch (const std::exception&) {
    }
  }
  if (begin < n) fn(begin, n);
}

}  // namespace ptyb::eng

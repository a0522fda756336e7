// Host loops over independent pieces of a table that is built once.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

namespace tfgb {

// f(i) for i in [0, n), on up to sixteen threads when `work` (in elements) is
// worth starting them; on the calling thread alone when none can start.
template <typename F>
void parallel_for(int64_t n, int64_t work, const F& f) {
  const int64_t hw = std::max(1u, std::thread::hardware_concurrency());
  const int64_t threads = std::min<int64_t>({n, hw, 16, 1 + work / 8192});
  std::atomic<int64_t> next{0};
  auto run = [&] {
    for (int64_t i = next.fetch_add(1); i < n; i = next.fetch_add(1)) f(i);
  };
  std::vector<std::thread> team;
  for (int64_t t = 1; t < threads; ++t) {
    try {
      team.emplace_back(run);
    } catch (...) {
      break;
    }
  }
  run();
  for (std::thread& t : team) t.join();
}

}  // namespace tfgb

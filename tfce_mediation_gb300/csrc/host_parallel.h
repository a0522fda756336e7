// Host loops over independent pieces of a table that is built once.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <exception>
#include <thread>
#include <vector>

namespace tfgb {

// f(i) for i in [0, n), on up to sixteen threads as `work` (in list entries, of
// about 10 ns each) is worth starting them, about 50 us each beside a CUDA context: four
// from 49k entries on, seven for the 983k of an L7 surface (all sixteen took a
// tenth longer there); on the calling thread alone when none can start.  What f
// throws (out of memory) ends the loop and is thrown again on the calling thread.
template <typename F>
void parallel_for(int64_t n, int64_t work, const F& f) {
  const int64_t hw = std::max(1u, std::thread::hardware_concurrency());
  const int64_t threads = std::min<int64_t>({n, hw, 16, std::min<int64_t>(4, 1 + work / 16384) + work / 262144});
  std::atomic<int64_t> next{0};
  std::atomic<bool> failed{false};
  std::exception_ptr thrown;
  auto run = [&] {
    try {
      for (int64_t i = next.fetch_add(1); i < n && !failed; i = next.fetch_add(1)) f(i);
    } catch (...) {
      if (!failed.exchange(true)) thrown = std::current_exception();
    }
  };
  std::vector<std::thread> team;
  try {
    team.reserve(std::max<int64_t>(threads, 1) - 1);
    for (int64_t t = 1; t < threads; ++t) team.emplace_back(run);
  } catch (...) {  // fewer then
  }
  run();
  for (std::thread& t : team) t.join();
  if (thrown) std::rethrow_exception(thrown);
}

}  // namespace tfgb

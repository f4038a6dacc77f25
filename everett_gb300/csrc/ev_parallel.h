// ev_parallel.h -- host work spread over a few threads.
#pragma once

#include <algorithm>
#include <cstdint>
#include <thread>
#include <vector>

namespace ev {

// f(i) for every i < count, on at most max_threads threads, the caller's
// among them, and on no more than there are indices.  A call for few indices
// starts few threads: planning a batch of 2 or 3 circuits on 16 new threads
// took 4.4 ms with four server workers doing so at once (0.1 here), nearly
// all of it thread starts.
template <typename F>
void parallel_for(uint64_t count, unsigned max_threads, F f) {
  const uint64_t n = std::min<uint64_t>(count, std::max(1u, max_threads));
  auto share = [&](uint64_t w) {
    for (uint64_t i = w; i < count; i += n) f(i);
  };
  std::vector<std::thread> others;
  for (uint64_t w = 1; w < n; ++w) others.emplace_back(share, w);
  share(0);
  for (std::thread& t : others) t.join();
}

}  // namespace ev

// parallel_for (everett_gb300/csrc/ev_parallel.h): every index once, on no
// more threads than indices or than the limit, the caller's among them.
#include <cstdio>
#include <map>
#include <mutex>

#include "ev_parallel.h"

int main() {
  int bad = 0;
  for (uint64_t count : {0, 1, 2, 3, 15, 16, 17, 100, 1000})
    for (unsigned limit : {0u, 1u, 2u, 16u}) {
      std::mutex mu;
      std::vector<int> runs(count, 0);
      std::map<std::thread::id, int> threads;
      ev::parallel_for(count, limit, [&](uint64_t i) {
        std::lock_guard<std::mutex> lock(mu);
        ++runs[i];
        ++threads[std::this_thread::get_id()];
      });
      const uint64_t most = std::min<uint64_t>(count, limit ? limit : 1);
      bool ok = threads.size() == most && (count == 0 || threads.count(std::this_thread::get_id()));
      for (int r : runs) ok = ok && r == 1;
      if (!ok) std::printf("count %llu limit %u: %zu threads\n", (unsigned long long)count, limit, threads.size());
      bad += !ok;
    }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}

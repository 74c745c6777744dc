// Eight threads reserve ranges of mixed lengths (falconnpp_b200/csrc/fpp_arena.h)
// until nothing fits: no two ranges may overlap, and none may end past the
// capacity.  Prints "ok <ranges>" or the first fault.  Built and run by
// tests/test_arena.py.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>

#include "fpp_arena.h"

int main() {
  long long total = 0;
  for (int round = 0; round < 200; ++round) {
    const unsigned cap = 20000;
    std::atomic<unsigned> used{0};
    std::atomic<int> ready{0};
    std::vector<std::vector<std::pair<unsigned, unsigned>>> got(8);
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
      th.emplace_back([&, t] {
        std::mt19937 rng(round * 8 + t);
        ready.fetch_add(1);
        while (ready.load() < 8) std::this_thread::yield();
        for (int i = 0; i < 400; ++i) {  // long ranges that fail beside short ones that fit
          const unsigned want = rng() % 4 ? 1 + rng() % 30 : 1 + rng() % 3000;
          const bool pause = rng() % 4 == 0;  // let others in between this one's steps
          const unsigned at = fpp::arena_reserve(
              want, cap, [&] { return used.load(); },
              [&](unsigned v) {
                const unsigned was = used.fetch_add(v);
                if (pause) std::this_thread::yield();
                return was;
              });
          if (at != fpp::kArenaFull) got[t].push_back({at, want});
        }
      });
    for (auto& x : th) x.join();
    std::vector<std::pair<unsigned, unsigned>> all;
    for (auto& g : got) all.insert(all.end(), g.begin(), g.end());
    std::sort(all.begin(), all.end());
    unsigned end = 0;
    for (auto& r : all) {
      if (r.first < end || r.second > cap || r.first > cap - r.second) {
        std::printf("round %d: [%u, +%u) after %u\n", round, r.first, r.second, end);
        return 1;
      }
      end = r.first + r.second;
    }
    total += (long long)all.size();
  }
  std::printf("ok %lld\n", total);
  return 0;
}

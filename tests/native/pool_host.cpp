// Test harness: the library's host threads (rabbitbin_b200/csrc/host_pack.cpp) on many
// short jobs of changing part counts, from several callers.  Prints the jobs of which
// a part ran not exactly once before the call returned.  Not part of the library.
#include <cstdio>
#include <cstdlib>
#include <memory>

#include "../../rabbitbin_b200/csrc/host_pack.cpp"

int main(int argc, char **argv) {
  const int jobs = std::atoi(argv[1]), callers = std::atoi(argv[2]);
  std::atomic<long> bad{0};
  auto caller = [&](int seed) {
    std::unique_ptr<std::atomic<int>[]> hits(new std::atomic<int>[64]);
    uint32_t x = 12345u + (uint32_t)seed;
    for (int j = 0; j < jobs; ++j) {
      x = x * 1664525u + 1013904223u;
      const int parts = 1 + (int)(x >> 16) % (j & 1 ? 3 : 40);
      for (int i = 0; i < 64; ++i) hits[i].store(0);
      rbg::pool().run([&](int i) { hits[i].fetch_add(1); }, parts);
      for (int i = 0; i < 64; ++i)
        if (hits[i].load() != (i < parts)) {
          bad.fetch_add(1);
          break;
        }
    }
  };
  std::vector<std::thread> th;
  for (int c = 0; c < callers; ++c) th.emplace_back(caller, c);
  for (auto &t : th) t.join();
  std::printf("%ld\n", bad.load());
  return 0;
}

// Host build of claim_entries (exact-depth-peeling_b200/csrc/edp_device.cuh)
// for the CPU tests: `threads` threads claim the given lengths from one pool,
// each its own run of `each` lengths, and record what they were granted.
#include <cstdint>
#include <thread>
#include <vector>

#include "../../exact-depth-peeling_b200/csrc/edp_device.cuh"

extern "C" int64_t claims(int threads, int each, const int *lengths, int64_t capacity,
                          int64_t *starts) {
  unsigned long long counter = 0;
  std::vector<std::thread> pool;
  for (int t = 0; t < threads; ++t)
    pool.emplace_back([&, t] {
      for (int k = t * each; k < (t + 1) * each; ++k)
        starts[k] = edp::claim_entries(&counter, lengths[k], capacity);
    });
  for (auto &t : pool) t.join();
  return int64_t(counter);
}

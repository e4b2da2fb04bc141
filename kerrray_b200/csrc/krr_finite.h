// Host scans of double arrays for infinities and NaN.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

namespace krr_host {

// Every value finite: a branch-free pass over the exponent fields (vectorised by the host
// compiler; an early-exit isfinite loop ran at a fraction of the memory bandwidth).
inline bool all_finite(const double* x, size_t n) {
  constexpr uint64_t kExp = 0x7ff0000000000000ull;
  uint64_t bad = 0;
  for (size_t i = 0; i < n; ++i) {
    uint64_t b;
    std::memcpy(&b, x + i, 8);
    bad |= (uint64_t)((b & kExp) == kExp);
  }
  return bad == 0;
}

// all_finite over up to 16 host threads for large arrays (memory-bandwidth bound).  A thread that
// cannot be started leaves its share to the others: no exception reaches a C entry point.
inline bool all_finite_parallel(const double* x, size_t n) {
  const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  if (n < ((size_t)1 << 22) || hw == 1) return all_finite(x, n);
  const size_t per = (n + hw - 1) / hw;
  std::atomic<size_t> next{0};
  std::atomic<bool> ok{true};
  auto work = [&] {
    for (size_t a = next.fetch_add(per); a < n && ok.load(); a = next.fetch_add(per))
      if (!all_finite(x + a, std::min(per, n - a))) ok.store(false);
  };
  std::vector<std::thread> threads;
  try {
    threads.reserve(hw - 1);
    for (unsigned t = 1; t < hw; ++t) threads.emplace_back(work);
  } catch (...) {
  }
  work();
  for (auto& th : threads) th.join();
  return ok.load();
}

}  // namespace krr_host

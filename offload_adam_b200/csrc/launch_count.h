// Launch accounting: every wrapper that launches one of our kernels bumps this counter, so
// that a benchmark can report how many of our launches ran in a region.  Autograd's device
// threads launch without the interpreter lock, so the addition is atomic (relaxed: it orders
// nothing).
#pragma once
#include <atomic>

namespace oab {

extern std::atomic<unsigned long long> g_launch_count;
inline void count_launch(unsigned long long n = 1) { g_launch_count.fetch_add(n, std::memory_order_relaxed); }

}  // namespace oab

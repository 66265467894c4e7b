// Threads that count launches at the same time lose none.
#include <stdio.h>

#include <thread>
#include <vector>

#include "../../offload_adam_b200/csrc/launch_count.h"

std::atomic<unsigned long long> oab::g_launch_count{0};

int main() {
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([] {
      for (int i = 0; i < 1000000; ++i) oab::count_launch();
    });
  for (auto& t : threads) t.join();
  const unsigned long long n = oab::g_launch_count;
  printf("%llu\n", n);
  return n == 8000000ull ? 0 : 1;
}

// Host-only check of hash_slot (wn_exact.h): hashes reach every part of a table, also of one
// with more than 2^25 slots, and collide no more than random slots do. Built and run by
// tests/test_exact_plan.py; needs no GPU. Prints "ok" on success.
#include <cmath>
#include <cstdio>
#include <vector>

#include "wn_exact.h"

int main() {
  for (int bits : {10, 16, 25, 26, 28, 30}) {
    const uint32_t mask = (1u << bits) - 1;
    const long long n = bits < 22 ? 1ll << bits : 1ll << 22;
    std::vector<long long> part(64, 0);
    std::vector<bool> used(static_cast<size_t>(mask) + 1);
    long long distinct = 0;
    uint64_t x = 1;
    for (long long i = 0; i < n; ++i) {
      x = x * 6364136223846793005ull + 1442695040888963407ull;
      const uint32_t slot = wn::hash_slot(static_cast<uint32_t>(x >> 32), mask);
      ++part[static_cast<size_t>(slot) >> (bits - 6)];
      if (!used[slot]) ++distinct;
      used[slot] = true;
    }
    // 64 equal parts: each within 6 standard deviations of its share; at least as many
    // different slots as n random ones give in a table of n (0.632 n), less 2 %.
    for (long long c : part)
      if (c < n / 64.0 - 6 * std::sqrt(n / 64.0) || c > n / 64.0 + 6 * std::sqrt(n / 64.0)) {
        std::printf("2^%d slots: %lld of %lld hashes in one 64th\n", bits, c, n);
        return 1;
      }
    if (distinct < 0.61 * n) {
      std::printf("2^%d slots: %lld different ones of %lld\n", bits, distinct, n);
      return 1;
    }
  }
  std::printf("ok\n");
  return 0;
}

// Checks and packing of the caller's host arrays (device="cpu" and "gpu" entry points).
//
// One pass each, over spans of at least 1 MiB on up to four threads: what these calls
// spend is reading memory. The soup is written in spans of 4 MiB: what other cores wrote
// costs the copy to the device that follows more than they save (28,322 faces on two
// threads: 117 us and a call of 470 us behind it, on one 170 and 332). On a B200's host,
// general array operations before and now, us: the (9, nf) soup of 28,322 faces
// 200 -> 170, of 243,602 2,392 -> 377; the finite and
// range checks of 121,801 vertices and 243,602 faces 464 -> 149, comparing both with a
// copy 290 -> 210; 3,145,728 coordinates checked 1,015 -> 250.
#include <sched.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <system_error>
#include <thread>

#include "../../include/wn_b200.h"

namespace {

constexpr int64_t kSpanBytes = 1 << 20, kFillSpanBytes = 4 << 20;
constexpr int kMostThreads = 4;

int usable_threads() {
  cpu_set_t set;
  CPU_ZERO(&set);
  return sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
}

// f(lo, hi) over spans of [0, n), `bytes` of memory an item. A thread that cannot be
// started leaves its span to the caller's.
template <class F>
void over_spans(int64_t n, int64_t bytes, const F& f, int64_t span = kSpanBytes) {
  const int64_t want = n / std::max<int64_t>(1, span / bytes);
  const int parts = want < 2 ? 1 : static_cast<int>(std::min<int64_t>(
                                       std::min<int64_t>(want, kMostThreads), usable_threads()));
  if (parts < 2) {
    f(int64_t(0), n);
    return;
  }
  std::thread threads[kMostThreads];
  const int64_t step = (n + parts - 1) / parts;
  int started = 1;
  for (; started < parts; ++started) {
    const int64_t lo = std::min(n, step * started), hi = std::min(n, lo + step);
    try {
      threads[started] = std::thread([&f, lo, hi] { f(lo, hi); });
    } catch (const std::system_error&) {
      break;
    }
  }
  f(int64_t(0), std::min(n, step));
  if (started < parts) f(std::min(n, step * started), n);
  for (int k = 1; k < started; ++k) threads[k].join();
}

}  // namespace

extern "C" {

int wn_host_finite(const double* x, int64_t n) {
  std::atomic<int> bad{0};
  over_spans(n, 8, [&](int64_t lo, int64_t hi) {
    constexpr uint64_t kExponent = 0x7ff0000000000000ull;
    for (int64_t b = lo; b < hi; b += 4096) {
      const int64_t e = std::min(hi, b + 4096);
      uint64_t any = 0;
      for (int64_t i = b; i < e; ++i) {
        uint64_t u;
        std::memcpy(&u, x + i, 8);
        any |= (u & kExponent) == kExponent ? ~uint64_t(0) : 0;
      }
      if (any) {
        bad.store(1, std::memory_order_relaxed);
        return;
      }
    }
  });
  return bad.load() ? 0 : 1;
}

int wn_host_in_range(const int64_t* x, int64_t n, int64_t limit) {
  std::atomic<int> bad{0};
  over_spans(n, 8, [&](int64_t lo, int64_t hi) {
    const uint64_t top = static_cast<uint64_t>(limit) - 1;
    uint64_t any = 0;  // its sign bit: of x, or of (limit - 1) - x
    for (int64_t i = lo; i < hi; ++i) {
      const uint64_t u = static_cast<uint64_t>(x[i]);
      any |= u | (top - u);
    }
    if (any >> 63) bad.store(1, std::memory_order_relaxed);
  });
  return bad.load() ? 0 : 1;
}

int wn_host_same(const void* a, const void* b, int64_t bytes) {
  if (a == b) return 1;
  std::atomic<int> other{0};
  over_spans(bytes, 2, [&](int64_t lo, int64_t hi) {
    if (std::memcmp(static_cast<const char*>(a) + lo, static_cast<const char*>(b) + lo,
                    static_cast<size_t>(hi - lo)) != 0)
      other.store(1, std::memory_order_relaxed);
  });
  return other.load() ? 0 : 1;
}

int wn_host_soup(const double* V, int64_t nv, const int64_t* F, int64_t nf, double* tri) {
  std::atomic<int> bad{0};
  over_spans(nf, 96, [&](int64_t lo, int64_t hi) {
    for (int64_t b = lo; b < hi; b += 512) {  // a corner at a time: three rows are written
      const int64_t e = std::min(hi, b + 512);
      for (int c = 0; c < 3; ++c) {
        double *px = tri + 3 * c * nf, *py = px + nf, *pz = py + nf;
        for (int64_t f = b; f < e; ++f) {
          const int64_t i = F[3 * f + c];
          if (i < 0 || i >= nv) {
            bad.store(1, std::memory_order_relaxed);
            return;
          }
          px[f] = V[3 * i];
          py[f] = V[3 * i + 1];
          pz[f] = V[3 * i + 2];
        }
      }
    }
  }, kFillSpanBytes);
  return bad.load() ? WN_EINVAL : WN_OK;
}

}  // extern "C"

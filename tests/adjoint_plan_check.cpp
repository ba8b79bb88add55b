// Host-only check of plan_adjoint_edges_mixed: the partial sums of many edges and queries take
// no more than 8 GiB or what two waves of CTAs need, whichever is more. Built and run by
// tests/test_exact_plan.py against libwn_b200.so; needs no GPU (one resident CTA per SM is
// assumed without one, so the SM count stands for the resident CTAs). Prints "ok" on success.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "wn_adjoint.h"

int main() {
  const long long sizes[] = {1000, 100000, 1000000, 10000000, 100000000};
  const int slots = 740;  // five resident CTAs on 148 SMs
  for (long long ne : sizes)
    for (long long nq : sizes) {
      const wn::AdjointPlan p = wn::plan_adjoint_edges_mixed(ne, nq, slots);
      const double bytes = static_cast<double>(wn::adjoint_edges_mixed_scratch_bytes(p, ne, nq));
      // 24 bytes a query and range, 48 an edge and group, split for the smallest sum over two
      // waves; and the sorted copies of edges and queries.
      const double two = 2.0 * std::sqrt(2.0 * slots * 24.0 * 48.0 * ne * nq) + 400.0 * ne + 200.0 * nq;
      if (bytes > std::max(1.1 * two, 8.0 * (1 << 30))) {
        std::printf("%lld edges x %lld queries: %.1f GB, two waves %.1f\n", ne, nq, bytes / 1e9,
                    two / 1e9);
        return 1;
      }
    }
  std::printf("ok\n");
  return 0;
}

// Host check of the launch plans of the pair-kernel precompute (doi_b200/csrc/rte_store_plan.h, compiled by g++ from
// tests/test_store_plan_cpu.py): over every column height up to 1024, grids of both precisions whose chosen layout
// does not fit the shared memory of a CTA.  Prints "plans <n> staged <n> over <n>".
#include <cstdio>

#include "rte_store_plan.h"

int main() {
  const size_t smem = 232448;  // opt-in limit of an sm_100 CTA
  long plans = 0, staged = 0, over = 0;
  for (int nz = 1; nz <= 1024; ++nz)
    for (int f = 0; f < 2; ++f) {
      auto one = [&](int nx, int ny) {
        if ((long long)nx * ny * nz > (1ll << 26)) return;
        const StPlan p = st_plan(nx, ny, nz, f != 0, smem);
        ++plans;
        staged += p.stage;
        over += p.bytes > smem || p.npair < st_pairs_per_lane(f != 0, p.stage);
      };
      // every number of columns whose mu_t shared memory could hold (as one row and as two), some beyond
      for (int n = 1; (long long)n * nz <= 60000 && n <= 1024; ++n) one(n, 1), one(n, n);
      for (int n = 1; (long long)n * n * nz <= 60000; ++n)
        for (int m = n; m <= n + 3; ++m) one(n, m);
      one(1024, 64), one(64, 1024), one(200, 200), one(1024, 1024);
    }
  std::printf("plans %ld staged %ld over %ld\n", plans, staged, over);
  return over ? 1 : 0;
}

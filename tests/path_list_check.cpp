// Host check of the closed-form path lists in doi_b200/csrc/rte_walk.cuh (compiled by g++ from tests/test_path_list_cpu.py)
// against a sequential walk: every displacement up to 12 and random ones up to 1023 with a product below 2^26, among
// them equal and commensurable ones (ties).  Each entry has to be made once, by one lane, with the walk's steps, length
// and leaving mark.  Prints "lists <n> entries <n> ties <n> mismatches <n>".
#include <cstdio>
#include <random>
#include <vector>

#include "rte_walk.cuh"

static long lists = 0, entries = 0, ties = 0, bad = 0;

static void check(int Dx, int Dy, int Dz) {
  const int mx = std::max(Dx, 1), my = std::max(Dy, 1), mz = std::max(Dz, 1), S = Dx + Dy + Dz;
  const long hx = (long)my * mz, hy = (long)mx * mz, hz = (long)mx * my, Q = 2l * mx * my * mz;
  struct E { int x, y, z; long len; bool leaves; };
  std::vector<E> want;
  long prev = 0;
  int cx = 0, cy = 0, cz = 0;
  for (int s = 0; s < S; ++s) {
    const long big = 1l << 60, ax = cx < Dx ? (2l * cx + 1) * hx : big, ay = cy < Dy ? (2l * cy + 1) * hy : big,
               az = cz < Dz ? (2l * cz + 1) * hz : big, m = std::min(ax, std::min(ay, az));
    ties += (ax == m) + (ay == m) + (az == m) > 1;
    const bool z = az == m, y = !z && ay == m;
    want.push_back({cx, cy, cz, m - prev, !z});
    prev = m;
    z ? ++cz : (y ? ++cy : ++cx);
  }
  want.push_back({cx, cy, cz, Q - prev, false});
  std::vector<int> made(S + 1, 0);
  for (int lane = 0; lane < 32; ++lane)
    path_list(Dx, Dy, Dz, lane, [&](int k, int x, int y, int z, int len, bool leaves) {
      if (k < 0 || k > S) {
        ++bad;
        return;
      }
      const E& w = want[k];
      ++made[k];
      if (x != w.x || y != w.y || z != w.z || len != w.len || leaves != w.leaves) ++bad;
    });
  for (int m : made) bad += m != 1;
  ++lists;
  entries += S + 1;
}

int main() {
  for (int x = 0; x <= 12; ++x)
    for (int y = 0; y <= 12; ++y)
      for (int z = 0; z <= 12; ++z) check(x, y, z);
  std::mt19937 rng(7);
  for (int t = 0; t < 4000; ++t) {
    int d[3];
    do
      for (int& q : d) q = (int)(rng() % (1u << (1 + rng() % 10))), q = q > 1023 ? 1023 : q;
    while ((long)std::max(d[0], 1) * std::max(d[1], 1) * std::max(d[2], 1) > (1l << 26));
    if (t % 4 == 0) d[1] = d[0];
    if (t % 8 == 0 && d[0]) d[2] = std::min(1023, d[2] / d[0] * d[0]);
    if ((long)std::max(d[0], 1) * std::max(d[1], 1) * std::max(d[2], 1) > (1l << 26)) continue;
    check(d[0], d[1], d[2]);
  }
  for (int q = 0; q < 3; ++q) check(q == 0 ? 1023 : 0, q == 1 ? 1023 : 0, q == 2 ? 1023 : 63);
  check(1023, 1023, 63);
  std::printf("lists %ld entries %ld ties %ld mismatches %ld\n", lists, entries, ties, bad);
  return bad ? 1 : 0;
}

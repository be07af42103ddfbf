// Shared memory of the pair-kernel precompute and the choice of its launch (host and device; no CUDA calls, so that the
// CPU tests evaluate it).
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define RTE_PLAN_FN __host__ __device__
#else
#define RTE_PLAN_FN
#endif

constexpr size_t ST_SMALL = 72 * 1024;  // shared memory of a CTA, three per SM
constexpr size_t ST_LARGE = 110 * 1024; // ... two per SM
constexpr int ST_PAIRS = 30;            // most column pairs of a chunk (a warp lays them out)
constexpr int ST_CAP = 3072;            // list entries per batch (one list has at most 3 * 1023 + 1)

// path sums per lane, of E column pairs: one list entry serves them all (33^3 FP32, mu_t in shared memory: 4 per lane
// 10.1 ms, 6 9.2; 41^3 through L1: 4 50 ms, 6 55)
RTE_PLAN_FN constexpr int st_pairs_per_lane(bool fp64, bool stage) { return !fp64 && stage ? 6 : 4; }

// bytes of a list entry (rte_store.cu): packed FP32 form, else column offset, z and length apart
RTE_PLAN_FN constexpr size_t st_entry_bytes(bool fp64, bool pack) { return !fp64 && pack ? 8 : 16; }

// entries [cap] | tile [npair][zb][zb | 1] | per list: f1, f2 | per pair and z: kernel offset of the destination and of the
// source column's position | per list: start | per pair: destination, source column | mu_t
struct StLayout {
  size_t off_tile, off_f, off_o, off_s, off_c, off_mu, bytes;
  RTE_PLAN_FN StLayout(size_t esize, size_t entry, int npair, int zb, int nz, int cap, int n_mu) {
    off_tile = entry * cap;
    off_f = (off_tile + esize * npair * zb * (zb | 1) + 15) / 16 * 16;
    off_o = off_f + esize * 2 * nz;
    off_s = off_o + sizeof(size_t) * 2 * npair * zb;
    off_c = off_s + sizeof(int) * nz;
    off_mu = (off_c + sizeof(int) * (2 * npair + 2) + 15) / 16 * 16;
    bytes = off_mu + esize * n_mu;
  }
};

struct StPlan {
  bool stage, pack;  // mu_t in shared memory; packed list entries
  int threads, npair, zb, cap;
  size_t bytes;
};

// Threads of a CTA: 256 with mu_t in shared memory and room for three CTAs per SM, which go through their barriers
// independently, else 512 (17^3 FP32 270 us with one CTA of 512 and chunks of 12 pairs in fixed turns; 200 with 256
// threads and units by a counter; 180 with chunks of up to 30; 152 with room for the entries the grid can have,
// FP64 442 -> 273).
inline StPlan st_plan(int nx, int ny, int nz, bool fp64, size_t smem) {
  StPlan p;
  const int N = nx * ny * nz, nblk = (nz + 47) / 48;
  const size_t es = fp64 ? 8 : 4;
  p.zb = (nz + nblk - 1) / nblk;
  // list entries of a batch: those of all lists of the longest displacement, when they are fewer
  const long long all = (long long)nz * (nx + ny - 1) + (long long)nz * (nz - 1) / 2;
  p.cap = (int)((all + 3) / 4 * 4 < ST_CAP ? (all + 3) / 4 * 4 : ST_CAP);
  auto bytes = [&](bool stage, bool pack, int npair) {
    return StLayout(es, st_entry_bytes(fp64, pack), npair, p.zb, nz, p.cap, stage ? N : 0).bytes;
  };
  // mu_t in shared memory when 48 KB and more remain for tiles beside the lists, and the least chunk fits: tiles of a z
  // block near 48 take 56 KB (FP32) or 75 KB (FP64)
  p.stage = es * N + p.cap * st_entry_bytes(fp64, true) + 48 * 1024 <= smem &&
            bytes(true, true, st_pairs_per_lane(fp64, true)) <= smem;
  p.pack = !fp64 && (p.stage || N < (1 << 21));
  const int E = st_pairs_per_lane(fp64, p.stage);
  p.threads = p.stage && bytes(true, p.pack, 2 * E) <= ST_SMALL ? 256 : 512;
  const size_t budget = p.threads == 256 ? ST_SMALL : p.stage && bytes(true, p.pack, 8) > ST_LARGE ? smem : ST_LARGE;
  p.npair = E;
  while (p.npair + E <= ST_PAIRS && bytes(p.stage, p.pack, p.npair + E) <= budget) p.npair += E;
  p.bytes = bytes(p.stage, p.pack, p.npair);
  return p;
}

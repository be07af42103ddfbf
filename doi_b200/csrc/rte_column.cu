// rte_column.cu -- the off-diagonal attenuation operator by voxel columns.
//
// The pair operator is out[r] = sum_r' R(w) k(r,r') (R(w) . W[r']), w the direction from r' to r.  All
// pairs of one destination column and one source column (fixed dx, dy) share the azimuth phi of w, and on
// that meridian every spherical harmonic of order <= L is a trigonometric polynomial in the polar angle
// theta alone:
//   R_lm(theta, phi) = N_lm U_lm(theta) (cos m phi | sin m phi),
//   U_lm = sum_k a_lmk cos k theta (m even) or sum_k a_lmk sin k theta (m odd), k <= l, k = l mod 2,
// so the (L+1)^2 source coefficients contract to 2L+1 numbers b_k once per (source, destination column),
// a pair costs 2L+1 multiply-adds in (S = sum_k b_k trig_k(theta)) and 2L+1 out (g_k += K S trig_k), and
// the sums g_k of one source column expand to the (L+1)^2 destination coefficients once per column pair:
// 22 multiply-adds per pair and right-hand side at L = 5 instead of 72, and no SH recurrence per pair.
// The trigonometric values come from (cos theta, sin theta) per displacement, tabulated in FP64 once per
// context (rte_launch_col_table), by double-angle and addition steps; for FP32 sums at L >= 7 they are FP64 values
// rounded: the whole row cos k theta, sin k theta is tabulated, or, in columns too long for that, made in FP64 from
// the FP64 pair.  (The contraction onto them is FP32 there too.  Against FP64, 25^3 L=7, six terms: 1.5e-7 with the
// kernel stored; per-pair functions evaluated in FP64, 6.5e-7 stored and 2.0e-7 recomputed, there 2.3e-7 now.)  The reference's snapped direction table (FisherInfo_IO) fits the
// same form: its azimuth index depends on (dx, dy) alone.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "rte_device.cuh"
#include "rte_internal.h"
#include "rte_trig.cuh"

namespace {

constexpr int T_CTA = 128;  // threads per CTA
#define RTE_FULL_L 7        // FP32 orders whose trigonometric rows are tabulated whole (FP64 values rounded)
#define RTE_FULL_NZ 512     // ... in columns of at most this many voxels

template <int N, typename F>
__device__ __forceinline__ void for_each_u(F f) {
  if constexpr (N > 0) {
    for_each_u<N - 1>(f);
    f(std::integral_constant<int, N - 1>{});
  }
}

// sources per stage of the kernel-value ring (a multiple of G), and its stages
template <int G>
__host__ __device__ constexpr int ring_rows() {
  return G == 3 ? 6 : 4;
}
template <int G>
__host__ __device__ constexpr int ring_stages() {
  return G == 3 ? 2 : 4;
}

// Shared memory (elements of T): [NB][tz][pitch] source rows | [2][ncd][azn] azimuth values | [ncd][polar]
// polar values | [ncd][tz][NB][nb_row] contracted sources | [4 warps][stages][rows][32 G] kernel values |
// 2 + 4 * stages mbarriers | the tensor-memory address, (x, y) of the destination columns
struct ColLayout {
  int off_a, off_t, off_b, off_k;
  size_t off_bar, off_xy, bytes;
  __host__ __device__ ColLayout(int tz, int pitch, int azn, int polar, int ncd, int nbr, int nb, int ring, int stages,
                                int esize) {
    off_a = nb * tz * pitch;
    off_t = off_a + 2 * ncd * azn;
    off_b = off_t + ncd * polar;
    off_k = off_b + ncd * tz * nbr;
    off_bar = ((size_t)(off_k + T_CTA / 32 * ring) * esize + 15) / 16 * 16;
    off_xy = off_bar + (2 + T_CTA / 32 * stages) * sizeof(uint64_t);
    bytes = off_xy + (1 + ncd) * sizeof(int);
  }
};

// columns of tensor memory for the sums of a thread's destinations (a power of two, at least 32)
template <int L, typename T, int G, int NB>
__host__ __device__ constexpr int tmem_cols() {
  int n = 32;
  while (n < NB * G * (L + 1) * (L + 1) * (int)(sizeof(T) / 4)) n *= 2;
  return n;
}

// One CTA: 128 threads of G consecutive destinations of a column each, against the source columns of its
// chunk, one run of tz sources of a column at a time.  What bounds it is the FMA pipe and, close behind, the shared memory's 128 bytes per
// cycle: a value read by every lane of a warp costs as much as 32 different ones, so the contracted source row
// (2L+1 numbers) is read once for G destinations, and since their displacements to consecutive sources overlap,
// one new trigonometric row per source serves all G.  The pair kernel is streamed by bulk copies, a ring of
// stages per warp (each warp's values are contiguous: kmat_index); register prefetch in its place waited on
// every load (5.9 ms against 2.7 at 33^3 L=5).  The coefficient sums, touched once per source column, live in
// tensor memory, which leaves the registers of four CTAs per SM (at 33^3 L=5 the
// layout's 58 KB admit three).  NB = 2: two right-hand sides a thread, which
// share the trigonometric rows, the kernel values and the copies (two CTAs per SM at L >= 4).  CPLX: (real, imaginary) rows of one complex
// right-hand side, the pair kernel times exp(-i kappa r) (phase tabulated beside the angles).
// 33^3 L=5 launch, FP32, one right-hand side: 7.40 ms by per-pair spherical harmonics -> 2.37; four: 20.1 -> 9.3, two a
// thread 8.2; FP64: 24.7 -> 4.2.  Of the 2.4 ms, skipping phases one at a time: pair loop 1.15, contraction 0.25, angle rows
// 0.2, the kernel stream 0.15, the rest expansion, start of runs and barriers.  All copies are bulk copies by warp 0
// and by each warp for its own ring (copies by all threads: 2.40, FP64 5.4); deeper rings and a fifth of the
// registers less did not pay (ring of 3 stages 2.37, four CTAs with 3-row stages 2.50).
template <int L, typename T, int G, int NB, bool CPLX, bool FULL>
__device__ __forceinline__ void column_body(const ColArgs& a) {
  constexpr int C = (L + 1) * (L + 1), NT = nb_row<L>(), LL = L > 0 ? L : 1;
  constexpr bool SUB = G == 1;  // one destination of each thread of the layout's groups
  constexpr bool F32 = std::is_same<T, float>::value;
  constexpr int U = ring_rows<G>(), NST = ring_stages<G>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ColLayout Sh(a.tz, a.pitch, a.azn, a.row - a.azn, a.ncd, NB * NT, NB, NST * U * 32 * G, NST, (int)sizeof(T));
  T* sW = reinterpret_cast<T*>(smem_raw);
  T* sA = sW + Sh.off_a;
  T* sT = sW + Sh.off_t;
  T* sB = sW + Sh.off_b;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + Sh.off_bar);
  uint32_t* stm = reinterpret_cast<uint32_t*>(smem_raw + Sh.off_xy);
  int* sxy = reinterpret_cast<int*>(stm + 1);
  const int wid = threadIdx.x / 32, lane = threadIdx.x % 32;
  T* sK = sW + Sh.off_k + wid * NST * U * 32 * G;
  uint64_t* kbar = bar + 2 + wid * NST;
  const int tid = threadIdx.x, nz = a.nz, ncol = a.nx * a.ny;
  const int nrg = CPLX ? 1 : a.nrhs / NB;  // groups of right-hand sides
  const int tile = blockIdx.x / nrg, rhs = (blockIdx.x - tile * nrg) * NB;
  const int p0 = tile * T_CTA * G, np = ncol * a.nzp;  // destination positions: columns padded to nzp
  // destination columns of the CTA (SUB: those of the layout's blocks that its warps lie in)
  const int pa = SUB ? p0 / (32 * a.group) * 32 * a.group : p0;
  const int pb = SUB ? ((p0 + T_CTA - 1) / (32 * a.group) + 1) * 32 * a.group : p0 + T_CTA * G;
  const int c0 = pa / a.nzp, ncd = (min(pb, np) - 1) / a.nzp - c0 + 1;
  const int pw = tile * (T_CTA / 32) + wid, pt = SUB ? (pw / a.group * 32 + lane) * a.group + pw % a.group : p0 + tid * G;
  const int p = min(pt, np - G);
  const bool act = pt < np;
  const int cd = p / a.nzp, z = p - cd * a.nzp, j = cd - c0;
  if (tid == 0) {
    mbar_init(&bar[0], 1);  // a run's source rows and azimuth values
    mbar_init(&bar[1], 1);  // its polar values
    for (int q = 0; q < T_CTA / 32 * NST; ++q) mbar_init(&bar[2 + q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid < 4 && a.red) a.red[tid] = 0.0;
  constexpr int TMC = tmem_cols<L, T, G, NB>(), W32 = sizeof(T) / 4;
  __syncwarp();
  if (wid == 0) tmem_alloc(stm, TMC);
  tmem_fence_before();
  for (int q = tid; q < ncd; q += T_CTA) sxy[q] = ((c0 + q) / a.nx) << 16 | (c0 + q) % a.nx;
  __syncthreads();
  tmem_fence_after();
  // this CTA's sources; none from rows too far from all of its destinations (rte_store.cu).  Read back from shared memory:
  // derived from c0 they cost 48 more bytes of spills at L = 7 (25^3, four right-hand sides 4.57 ms a launch, 4.46 here)
  const int cb = max(a.col0 + (int)blockIdx.y * a.chunk, ((sxy[0] >> 16) - a.ry) * a.nx);
  const int ce = min(min(a.col1, a.col0 + ((int)blockIdx.y + 1) * a.chunk), ((sxy[ncd - 1] >> 16) + a.ry + 1) * a.nx);
  const int nrun = (nz + a.tz - 1) / a.tz, ntile = max(ce - cb, 0) * nrun;
  const uint32_t tm = *stm + ((uint32_t)(wid * 32) << 16);  // this warp's lanes, column 0
  const T* gW = static_cast<const T*>(a.W) + (size_t)rhs * a.N * a.pitch;
  const T* gT = static_cast<const T*>(a.tab);
  // kernel values of this warp's destinations: rows of 32 * group per source slot
  const int kb = 32 * a.group;
  const T* gK = static_cast<const T*>(a.K) +
                ((size_t)(SUB ? pw / a.group : pw) * a.Kld) * kb + (SUB ? pw % a.group * 32 : 0);
  const bool wact = (SUB ? pw / a.group * kb : pw * kb) < np;  // warps beyond the last block have no rows
  // a run: sources z0 .. z0 + tz of column col; the runs of a column follow one another
  struct Run {
    int col, xs, ys, z0;
  };
  auto after = [&](Run r) {
    r.z0 += a.tz;
    if (r.z0 >= nz) {
      r.z0 = 0;
      ++r.col;
      if (++r.xs == a.nx) r.xs = 0, ++r.ys;
    }
    return r;
  };
  // Copies by warp 0.  A run's source rows (one buffer, free after its contraction) and azimuth values (buffer b)
  // come while the previous run's pairs are summed, its polar values (one buffer) while it is contracted.
  auto angle_row = [&](const Run& r, int jj) {
    const int xd = sxy[jj] & 0xffff, yd = sxy[jj] >> 16;
    return gT + ((size_t)(yd - r.ys + a.ny - 1) * (2 * a.nx - 1) + (xd - r.xs + a.nx - 1)) * a.row;
  };
  const uint32_t azb = (uint32_t)(a.azn * sizeof(T)), pob = (uint32_t)((a.row - a.azn) * sizeof(T));
  auto rows = [&](const Run& r, int b) {
    const int ns = min(a.tz, nz - r.z0), s0 = r.col * nz + r.z0;
    const uint32_t bw = (uint32_t)(ns * a.pitch * sizeof(T));
    if (lane == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&bar[0], NB * bw + ncd * azb);
#pragma unroll
      for (int q = 0; q < NB; ++q) bulk_g2s(sW + q * a.tz * a.pitch, gW + ((size_t)q * a.N + s0) * a.pitch, bw, &bar[0]);
    }
    __syncwarp();
    if (azb > 0)
      for (int jj = lane; jj < ncd; jj += 32) bulk_g2s(sA + (b * a.ncd + jj) * a.azn, angle_row(r, jj), azb, &bar[0]);
  };
  auto polars = [&](const Run& r) {
    if (lane == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&bar[1], ncd * pob);
    }
    __syncwarp();
    for (int jj = lane; jj < ncd; jj += 32)
      bulk_g2s(sT + jj * (a.row - a.azn), angle_row(r, jj) + a.azn, pob, &bar[1]);
  };
  // Ring of kernel values: groups of up to U sources (groups do not cross runs), one per stage.
  const T* k_src = gK + (size_t)(cb * nz - a.kslot0) * kb;  // cursor of the next group to copy
  int k_rem = max(ce - cb, 0) * nz, k_z = 0, k_left = min(a.tz, nz), k_st = 0, k_fly = 0;
  auto next_group = [&]() {
    if (k_rem <= 0) return;
    const int n = min(U, k_left);
    if (wact) {
      T* dst = sK + k_st * U * 32 * G;
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&kbar[k_st], (uint32_t)(n * 32 * G * sizeof(T)));
        if constexpr (!SUB) bulk_g2s(dst, k_src, (uint32_t)(n * 32 * G * sizeof(T)), &kbar[k_st]);
      }
      if constexpr (SUB) {
        __syncwarp();
        if (lane < n) bulk_g2s(dst + lane * 32, k_src + (size_t)lane * kb, 32 * sizeof(T), &kbar[k_st]);
      }
    }
    ++k_fly;
    k_src += n * kb;
    k_rem -= n;
    k_left -= n;
    if (k_left == 0) {  // the next run
      k_z = k_z + a.tz < nz ? k_z + a.tz : 0;
      k_left = min(a.tz, nz - k_z);
    }
    if (++k_st == NST) k_st = 0;
  };
  int u_st = 0;  // stage of the next group to use, and its phase
  uint32_t u_ph = 0;
  bool kok = true;
  {  // the destinations' coefficient sums live in tensor memory, one row of C values per destination
    uint32_t zero[C * W32];
#pragma unroll
    for (int c = 0; c < C * W32; ++c) zero[c] = 0u;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB * G; ++i) tmem_st<C * W32>(tm + i * C * W32, zero);
    tmem_wait_st();
  }
  Run cur{cb, cb % a.nx, cb / a.nx, 0};
  if (ntile > 0) {
    if (wid == 0) {
      rows(cur, 0);
      polars(cur);
    }
    for (int q = 0; q < NST; ++q) next_group();
  }
  const int nmag = ((1 << 22) + min(a.tz, nz) - 1) / min(a.tz, nz);  // q / tz = q * nmag >> 22 (q * tz < 2^22)
  for (int t = 0; t < ntile; ++t) {
    const int bf = t & 1;
    const Run nxt = after(cur);
    const bool ok = mbar_wait(&bar[0], (uint32_t)bf);
    if (__syncthreads_or(!ok || !kok)) {
      if (tid == 0) {
        atomicExch(a.err, 1);
        mbar_wait(&bar[1], (uint32_t)bf);  // copies in flight
      }
      for (; wact && k_fly > 0; --k_fly) {
        mbar_wait(&kbar[u_st], u_ph);
        if (++u_st == NST) u_st = 0, u_ph ^= 1;
      }
      tmem_fence_before();
      __syncthreads();
      tmem_fence_after();
      __syncwarp();
      if (wid == 0) tmem_free(*stm, TMC);
      return;
    }
    const int z0 = cur.z0, ns = min(a.tz, nz - z0);
    const T* At = sA + bf * a.ncd * a.azn;
    // contract the run's sources onto the destination columns' meridians, two columns per row read
    // (neighbouring threads take neighbouring sources: rows are an odd number of 16-byte units apart, so the
    // loads are conflict-free)
    for (int q = tid; q < (ncd + 1) / 2 * NB * a.tz; q += T_CTA) {
      const int jb = (int)(((long long)q * nmag) >> 22), s = q - jb * a.tz, jp = jb / NB, b = jb - jp * NB;
      if (s >= ns) continue;
      const T* w = sW + (b * a.tz + s) * a.pitch;
      T row[C];
      if constexpr (F32) {
#pragma unroll
        for (int c = 0; c < up4(C); c += 4) {
          const float4 v = *reinterpret_cast<const float4*>(w + c);
          row[c] = v.x;
          if (c + 1 < C) row[c + 1] = v.y;
          if (c + 2 < C) row[c + 2] = v.z;
          if (c + 3 < C) row[c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < C; c += 2) {
          const double2 v = *reinterpret_cast<const double2*>(w + c);
          row[c] = v.x;
          if (c + 1 < C) row[c + 1] = v.y;
        }
      }
#pragma unroll 1
      for (int jj = 2 * jp; jj < min(2 * jp + 2, ncd); ++jj) {
        T bq[NT];
        contract_row<L, T>(row, At + jj * a.azn, bq);
        T* d = sB + ((jj * a.tz + s) * NB + b) * NT;
        if constexpr (F32) {
#pragma unroll
          for (int c = 0; c < NT; c += 4)
            *reinterpret_cast<float4*>(d + c) = make_float4(bq[c], bq[c + 1], bq[c + 2], bq[c + 3]);
        } else {
#pragma unroll
          for (int c = 0; c < NT; c += 2) *reinterpret_cast<double2*>(d + c) = make_double2(bq[c], bq[c + 1]);
        }
      }
    }
    __syncthreads();
    if (wid == 0 && t + 1 < ntile) rows(nxt, bf ^ 1);
    kok = mbar_wait(&bar[1], (uint32_t)bf) && kok;
    const T* B = sB + j * a.tz * NB * NT;
    typedef typename std::conditional<F32, f2_t, double2>::type Pair;
    Pair tr[G][LL];  // p_k (signed) of destination i, source sb + u at slot (i - u) mod G
    [[maybe_unused]] T ph[CPLX ? G : 1][2];
    // angle entries lie by residue class of their index e = dz + nz modulo G (lanes are G apart, so a warp reads
    // neighbouring entries): ap[i] the next entry below of the class that step u = i (mod G) needs
    const T* ap[G];
    auto turn = [&](const T* an, int q) {  // trigonometric pairs of one displacement into slot q
      if constexpr (FULL) {
#pragma unroll
        for (int k = 0; k < L; ++k) tr[q][k] = reinterpret_cast<const f2_t*>(an)[k];
      } else if constexpr (F32 && L >= RTE_FULL_L) {
        double ck[L], sk[L];
        const double2 v = *reinterpret_cast<const double2*>(an);
        trig_pairs<L, double>(v.x, v.y, fma(v.x, v.x, -(v.y * v.y)), 2.0 * v.x * v.y, ck, sk);
#pragma unroll
        for (int k = 0; k < L; ++k) tr[q][k] = f2_pack((float)ck[k], (float)sk[k]);
      } else if constexpr (L > 0) {
        T ck[L], sk[L];
        if constexpr (F32) {
          const float4 v = *reinterpret_cast<const float4*>(an);
          trig_pairs<L, float>(v.x, v.y, v.z, v.w, ck, sk);
#pragma unroll
          for (int k = 0; k < L; ++k) tr[q][k] = f2_pack(ck[k], sk[k]);
        } else {
          const double2 v = *reinterpret_cast<const double2*>(an);
          trig_pairs<L, double>(v.x, v.y, fma(v.x, v.x, -(v.y * v.y)), 2.0 * v.x * v.y, ck, sk);
#pragma unroll
          for (int k = 0; k < L; ++k) tr[q][k] = make_double2(ck[k], sk[k]);
        }
      }
      if constexpr (CPLX) ph[q][0] = an[a.pho], ph[q][1] = an[a.pho + 1];
    };
    {
      const T* ang = sT + j * (a.row - a.azn);
      const int e0 = z - z0 + nz;
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int e = e0 + i, r = e % G;
        turn(ang + (r * a.cls + e / G) * a.csn, i);
        const int f = e0 - 1 - i, rf = f % G;  // f >= 0 while source i exists
        ap[i] = ang + (rf * a.cls + f / G) * a.csn;
      }
    }
    Pair g2[NB][G][LL];
    T g0[NB][G];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < G; ++i) {
        g0[b][i] = T(0);
#pragma unroll
        for (int k = 0; k < LL; ++k) {
          if constexpr (F32)
            g2[b][i][k] = 0ull;
          else
            g2[b][i][k] = make_double2(0.0, 0.0);
        }
      }
    auto step = [&](auto uc, int s, const T* Kt) {
      constexpr int u = decltype(uc)::value;
      T S[NB][G];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const T* w = B + (s * NB + b) * NT;
        if constexpr (F32) {
          f2_t wv[NT / 2];
#pragma unroll
          for (int c = 0; c < NT / 4; ++c) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(w)[c];
            wv[2 * c] = (f2_t)v.x;
            wv[2 * c + 1] = (f2_t)v.y;
          }
#pragma unroll
          for (int i = 0; i < G; ++i) {
            const int q = ((i - u) % G + G) % G;
            f2_t acc = wv[L];  // (b_0, 0)
#pragma unroll
            for (int k = 0; k < L; ++k) acc = f2_fma(tr[q][k], wv[k], acc);
            float lo, hi;
            f2_unpack(acc, lo, hi);
            S[b][i] = Kt[u * 32 * G + i * 32] * (lo + hi);
          }
        } else {
          double2 wv[LL];
#pragma unroll
          for (int k = 0; k < L; ++k) wv[k] = reinterpret_cast<const double2*>(w)[k];
          const double w0 = w[2 * L];
#pragma unroll
          for (int i = 0; i < G; ++i) {
            const int q = ((i - u) % G + G) % G;
            double s0 = w0, s1 = 0.0;
#pragma unroll
            for (int k = 0; k < L; ++k) {
              s0 = fma(tr[q][k].x, wv[k].x, s0);
              s1 = fma(tr[q][k].y, wv[k].y, s1);
            }
            S[b][i] = Kt[u * 32 * G + i * 32] * (s0 + s1);
          }
        }
      }
      if constexpr (CPLX) {  // (S0 + i S1) exp(-i kappa r)
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const int q = ((i - u) % G + G) % G;
          const T t0 = ph[q][0] * S[0][i] + ph[q][1] * S[NB - 1][i], t1 = ph[q][0] * S[NB - 1][i] - ph[q][1] * S[0][i];
          S[0][i] = t0;
          S[NB - 1][i] = t1;
        }
      }
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const int q = ((i - u) % G + G) % G;
          const T v = S[b][i];
          g0[b][i] += v;
          if constexpr (F32) {
            const f2_t v2 = f2_pack(v, v);
#pragma unroll
            for (int k = 0; k < L; ++k) g2[b][i][k] = f2_fma(tr[q][k], v2, g2[b][i][k]);
          } else {
#pragma unroll
            for (int k = 0; k < L; ++k) {
              g2[b][i][k].x = fma(tr[q][k].x, v, g2[b][i][k].x);
              g2[b][i][k].y = fma(tr[q][k].y, v, g2[b][i][k].y);
            }
          }
        }
      // the next source's new displacement z - (s + 1) takes the slot of the last destination
      turn(ap[u % G], ((G - 1 - u) % G + G) % G);
      ap[u % G] -= a.csn;
    };
    for (int sb = 0; sb < ns; sb += U) {
      if (wact) kok = mbar_wait(&kbar[u_st], u_ph) && kok;
      const T* Kt = sK + u_st * U * 32 * G + lane;
      if (++u_st == NST) u_st = 0, u_ph ^= 1;
      --k_fly;
      if (sb + U <= ns)
        for_each_u<U>([&](auto uc) { step(uc, sb + decltype(uc)::value, Kt); });
      else
        for_each_u<U - 1>([&](auto uc) {
          if (sb + decltype(uc)::value < ns) step(uc, sb + decltype(uc)::value, Kt);
        });
      __syncwarp();
      next_group();
    }
    __syncwarp();  // one lane's copies, a wait's end
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < G; ++i) {
        T g[NT];
        g[2 * L] = g0[b][i];
#pragma unroll
        for (int k = 0; k < L; ++k) {
          if constexpr (F32) {
            f2_unpack(g2[b][i][k], g[2 * k], g[2 * k + 1]);
          } else {
            g[2 * k] = g2[b][i][k].x;
            g[2 * k + 1] = g2[b][i][k].y;
          }
        }
        const uint32_t at = tm + (b * G + i) * C * W32;
        T out[C];
        tmem_ld<C * W32>(at, reinterpret_cast<uint32_t*>(out));
        tmem_wait_ld<C * W32>(reinterpret_cast<uint32_t*>(out));
        expand_row<L, T>(g, At + j * a.azn, out);
        tmem_st<C * W32>(at, reinterpret_cast<const uint32_t*>(out));
      }
    tmem_wait_st();
    cur = nxt;
    __syncthreads();  // the contracted sources and buffer bf are free for run t + 2
    if (wid == 0 && t + 1 < ntile) polars(cur);
  }
  if (!kok && lane == 0) atomicExch(a.err, 1);
#pragma unroll
  for (int i = 0; i < G; ++i)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      T out[C];
      __syncwarp();  // the branch of the previous destination (ragged columns, the last tile)
      tmem_ld<C * W32>(tm + (b * G + i) * C * W32, reinterpret_cast<uint32_t*>(out));
      tmem_wait_ld<C * W32>(reinterpret_cast<uint32_t*>(out));
      if (!act || z + i >= nz) continue;
      const size_t r = (size_t)(z + i) * ncol + cd;
      T* o = static_cast<T*>(a.part) + ((size_t)(a.split0 + blockIdx.y) * a.N + r) * a.vstride + (rhs + b) * a.Cfull;
      // chunk sums: FP32 as they are (the epilogue applies N_c after adding the chunks in FP64), FP64 times N_c
      if (F32 && C % 4 == 0 && a.Cfull % 4 == 0) {
#pragma unroll
        for (int c = 0; c + 3 < C; c += 4)
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(o) + c) =
              make_float4((float)out[c], (float)out[c + 1], (float)out[c + 2], (float)out[c + 3]);
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) o[c] = F32 ? out[c] : out[c] * (T)kMonic.N[c];
      }
    }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  __syncwarp();
  if (wid == 0) tmem_free(*stm, TMC);
}

// CTAs per SM to fit the registers to (shared memory may admit fewer, three at 33^3 L=5): their warps hide the latencies
// of one another's loads (33^3 L=5: 2.77 ms per launch at two CTAs with the sums in registers, 2.41 with them in tensor
// memory and the registers of four)
template <int L, typename T, int NB, bool CPLX>
__host__ __device__ constexpr int col_ctas() {
  if (CPLX || (NB == 2 && L >= 4)) return 2;
  if (NB == 2) return 3;
  return std::is_same<T, float>::value ? (L <= 5 ? 4 : 3) : (L <= 3 ? 2 : 1);
}

template <int L, typename T, int G, int NB, bool CPLX, bool FULL>
__global__ void __launch_bounds__(T_CTA, col_ctas<L, T, NB, CPLX>()) k_column(ColArgs a) {
  column_body<L, T, G, NB, CPLX, FULL>(a);
}

// Angle rows: per column displacement (dx, dy) first azn values (cos m phi, sin m phi, m = 1..L), then the polar
// entries of dz = e - nz, e = 0..nz+nzp-1, csn values each, entry e at (e % tg) * cls + e / tg: (cos theta,
// sin theta), for FP32 also (cos 2theta, sin 2theta), for FP32 at L >= 7 every (cos k theta, sin k theta) or, in long
// columns, (cos theta, sin theta) in FP64, and with kappa != 0 the phase (cos kappa r, sin kappa r) at offset pho.  One thread per (dx, dy, dz).
template <typename T>
__global__ void k_col_table(ColTabArgs a, T* tab) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int mz = a.nz + a.nzp, mx = 2 * a.nx - 1, my = 2 * a.ny - 1;
  if (t >= (long long)mx * my * mz) return;
  const int iz = (int)(t % mz), ix = (int)((t / mz) % mx), iy = (int)(t / ((long long)mz * mx));
  const int dx = ix - (a.nx - 1), dy = iy - (a.ny - 1), dz = iz - a.nz;
  T* row = tab + ((size_t)iy * mx + ix) * a.row;
  const double ex = dx * a.dx, ey = dy * a.dy, ez = dz * a.dz;
  const double rho = sqrt(ex * ex + ey * ey), r = sqrt(ex * ex + ey * ey + ez * ez);
  double cp = 1.0, sp = 0.0, ct = 1.0, st = 0.0;
  if (a.table) {  // the reference's cell (table_direction): theta index from dz, phi index from (dx, dy)
    const int sg = a.transpose ? -1 : 1;
    const double fx = (double)(sg * dx) * a.dx, fy = (double)(sg * dy) * a.dy, fz = (double)(sg * dz) * a.dz;
    int ti = r > 0.0 ? (int)rintf((float)((100 - 1) * (acos(fz / r)) / (M_PI))) : 0;
    const int pj = (int)rintf((float)((100 - 1) * (atan2(fy, fx)) / (2 * M_PI)));
    // a negative phi index reads the previous theta row (theta 0 stays at the pole, where phi is immaterial)
    if (pj < 0) ti = max(ti - 1, 0);
    sincos((ti * M_PI) / (100 - 1), &st, &ct);
    sincos(((pj < 0 ? 100 + pj : pj) * 2.0 * M_PI) / (100 - 1), &sp, &cp);
  } else {
    if (rho > 0.0) cp = ex / rho, sp = ey / rho;
    if (r > 0.0) ct = ez / r, st = rho / r;
  }
  if (iz == 0) {
    double cm = 1.0, sm = 0.0;
    for (int m = 1; m <= a.L; ++m) {
      const double n = cm * cp - sm * sp;
      sm = cm * sp + sm * cp;
      cm = n;
      row[2 * m - 2] = (T)cm;
      row[2 * m - 1] = (T)sm;
    }
    for (int q = 2 * a.L; q < a.azn; ++q) row[q] = T(0);
  }
  T* p = row + a.azn + ((size_t)(iz % a.tg) * a.cls + iz / a.tg) * a.csn;
  double c = 1.0, s = 0.0;
  if (a.wide) *reinterpret_cast<double2*>(p) = make_double2(ct, st);  // in the place of two FP32 pairs
  for (int k = 1; k <= (a.wide ? 0 : a.nk); ++k) {
    const double n = c * ct - s * st;
    s = c * st + s * ct;
    c = n;
    p[2 * k - 2] = (T)c;
    p[2 * k - 1] = (T)s;
  }
  if (a.pho > 0) {
    double sn, cs;
    sincos(a.kappa * r, &sn, &cs);
    p[a.pho] = (T)cs;
    p[a.pho + 1] = (T)sn;
  }
}

// voxel-order rows [N][nb][Cfull] -> column-order rows [nb][N][pitch], coefficient c times N_c
template <typename T>
__global__ void k_rows(const double* w, T* rows, const int* islot, int N, int nb, int pitch, int Cfull) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int vstride = nb * Cfull;
  if (t >= (long long)N * vstride) return;
  const int r = (int)(t / vstride), e = (int)(t % vstride);
  const int rhs = e / Cfull, c = e - rhs * Cfull;
  rows[((size_t)rhs * N + islot[r]) * pitch + c] = (T)(w[t] * kMonic.N[c]);
}

// Dynamic shared memory above 48 KB: the attribute is set to the device's opt-in maximum, the same value from every host
// thread, not to one launch's size: the server launches the same instantiation from several worker threads with sizes
// that depend on the context, and per-launch values let one thread lower the limit between another's set and launch.
cudaError_t smem_limit(const void* kern, size_t smem) {
  int dev = 0, cap = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (smem > (size_t)cap) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
}

template <int L, typename T, int G, int NB, bool CPLX>
cudaError_t launch_nb(ColArgs a, cudaStream_t st, int* occ) {
  void (*kern)(ColArgs) = k_column<L, T, G, NB, CPLX, false>;
  if constexpr (L >= RTE_FULL_L && std::is_same<T, float>::value)
    if (a.nz <= RTE_FULL_NZ) kern = k_column<L, T, G, NB, CPLX, true>;
  const int np = a.nx * a.ny * a.nzp;
  // positions a CTA's columns span: its threads' destinations, or (G = 1) the layout blocks of its warps
  const int span = G == 1 ? ((T_CTA / 32 + a.group - 2) / a.group + 1) * 32 * a.group : T_CTA * G;
  a.ncd = (span + a.nzp - 2) / a.nzp + 1;
  const int nblk = (np + 32 * a.group - 1) / (32 * a.group);  // layout blocks: a warp each, or `group` warps for G = 1
  const int warps = G == 1 ? nblk * a.group : nblk;
  dim3 grid((unsigned)((warps + T_CTA / 32 - 1) / (T_CTA / 32)) * (CPLX ? 1 : a.nrhs / NB), a.nsplit);
  // the whole column as one run when two CTAs fit an SM's shared memory, else equal runs; where the angle rows leave no
  // room for two CTAs at runs of 8, the shared memory of one and up to 64 sources (1x1x500 L=7 mixed, six terms and
  // the final application 3.8 ms in runs of 8 -> 3.2; FP32 sums of 512 sources 2.1e-7 from FP64, of 64 1.5e-7)
  auto bytes = [&](int tz) {
    return ColLayout(tz, a.pitch, a.azn, a.row - a.azn, a.ncd, NB * nb_row<L>(), NB,
                     ring_stages<G>() * ring_rows<G>() * 32 * G, ring_stages<G>(), (int)sizeof(T)).bytes;
  };
  size_t smem = 0;
  auto runs = [&](int nrun, size_t limit) {
    do {
      a.tz = (a.nz + nrun - 1) / nrun++;
      smem = bytes(a.tz);
    } while (smem > limit && a.tz > 8);
    return smem <= limit;
  };
  if (!runs(1, 113 * 1024)) runs((a.nz + 63) / 64, 227 * 1024);
  cudaError_t e = smem_limit((const void*)kern, smem);
  if (e != cudaSuccess) return e;
  if (occ) {  // by registers, shared and tensor memory (the runtime's query answers 1 for kernels that use the latter)
    cudaFuncAttributes at;
    e = cudaFuncGetAttributes(&at, (const void*)kern);
    if (e != cudaSuccess) return e;
    const size_t regs = (size_t)(at.numRegs * 32 + 255) / 256 * 256 * (T_CTA / 32);
    *occ = (int)std::min<size_t>(std::min<size_t>(65536 / regs, 228 * 1024 / (smem + 1024)), 512 / tmem_cols<L, T, G, NB>());
    return cudaSuccess;
  }
  kern<<<grid, T_CTA, smem, st>>>(a);
  return cudaGetLastError();
}

// Right-hand sides of a thread: RTE_COL_NB where the launch has an even number of real ones in FP32.
template <int L, typename T, int G, bool CPLX>
cudaError_t launch_one(const ColArgs& a, cudaStream_t st, int* occ) {
  if constexpr (CPLX) {
    return launch_nb<L, T, G, 2, true>(a, st, occ);
  } else {
    if constexpr (std::is_same<T, float>::value && RTE_COL_NB(L) == 2)
      if (a.nrhs % 2 == 0) return launch_nb<L, T, G, 2, false>(a, st, occ);
    return launch_nb<L, T, G, 1, false>(a, st, occ);
  }
}

// Destinations per thread: RTE_COL_G; a complex pair's kernel may take one on the same layout (RTE_COL_GC).  A launch of a lower
// order than the context's (l = 0 passes of isotropic scatter) runs on its layout, so order 0 takes any of them.
template <int L, int G, int GC, int GC64>
cudaError_t launch_G(const ColArgs& a, int fp64, int cplx, cudaStream_t st, int* occ) {
  if (cplx) return fp64 ? launch_one<L, double, GC64, true>(a, st, occ) : launch_one<L, float, GC, true>(a, st, occ);
  return fp64 ? launch_one<L, double, G, false>(a, st, occ) : launch_one<L, float, G, false>(a, st, occ);
}

template <int L>
cudaError_t launch_L(const ColArgs& a, int fp64, int cplx, cudaStream_t st, int* occ) {
  if constexpr (L == 0) {
    switch (a.tg) {
      case 1: return launch_G<0, 2, 1, 1>(a, fp64, cplx, st, occ);
      case 2: return launch_G<0, 2, 2, 2>(a, fp64, cplx, st, occ);
      default: return launch_G<0, 3, 3, 3>(a, fp64, cplx, st, occ);
    }
  } else {
    return launch_G<L, RTE_COL_G(L), RTE_COL_GC(L, 0), RTE_COL_GC(L, 1)>(a, fp64, cplx, st, occ);
  }
}

}  // namespace

ColDims rte_col_dims(int C, int L, int nz, int fp64, int cplx) {
  ColDims d;
  const int unit = fp64 ? 2 : 4;  // elements per 16 bytes
  d.pitch = (C + unit - 1) / unit * unit;
  if ((d.pitch / unit) % 2 == 0) d.pitch += unit;
  d.group = RTE_COL_G(L);
  d.nzp = (nz + d.group - 1) / d.group * d.group;
  d.azn = up4(2 * L);
  // FP32 at L >= 7 tabulates whole trigonometric rows, an odd number of 8-byte units apart (conflict-free);
  // columns so long that two of them no longer fit shared memory keep the FP64 pair in the place of two FP32 ones
  const bool full = !fp64 && L >= RTE_FULL_L && nz <= RTE_FULL_NZ;
  d.nk = fp64 ? 1 : (full ? L : 2);
  d.wide = !fp64 && L >= RTE_FULL_L && !full;
  d.pho = cplx ? 2 * d.nk : 0;
  d.csn = 2 * d.nk + (cplx ? (fp64 ? 2 : 4) : 0);
  d.tg = cplx ? RTE_COL_GC(L, fp64) : d.group;
  d.cls = (nz + d.nzp + d.tg - 1) / d.tg;
  d.row = (d.azn + d.tg * d.cls * d.csn + unit - 1) / unit * unit;
  return d;
}

int rte_col_reach(int nx, int nzp, int group, int ry) {
  const int ncd = (T_CTA * group + nzp - 2) / nzp + 1;  // columns of a CTA at most, and the rows they lie in
  return ry + (ncd + nx - 2) / nx;
}

cudaError_t rte_launch_column(const ColArgs& a, int LA, int fp64, int cplx, cudaStream_t st, int* occ) {
  switch (LA) {
    case 0: return launch_L<0>(a, fp64, cplx, st, occ);
    case 1: return launch_L<1>(a, fp64, cplx, st, occ);
    case 2: return launch_L<2>(a, fp64, cplx, st, occ);
    case 3: return launch_L<3>(a, fp64, cplx, st, occ);
    case 4: return launch_L<4>(a, fp64, cplx, st, occ);
    case 5: return launch_L<5>(a, fp64, cplx, st, occ);
    case 6: return launch_L<6>(a, fp64, cplx, st, occ);
    case 7: return launch_L<7>(a, fp64, cplx, st, occ);
  }
  return cudaErrorInvalidValue;
}

cudaError_t rte_launch_col_table(const ColTabArgs& a, void* tab, int fp64, cudaStream_t st) {
  const long long n = (long long)(2 * a.nx - 1) * (2 * a.ny - 1) * (a.nz + a.nzp);
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (fp64)
    k_col_table<double><<<blocks, 256, 0, st>>>(a, static_cast<double*>(tab));
  else
    k_col_table<float><<<blocks, 256, 0, st>>>(a, static_cast<float*>(tab));
  return cudaGetLastError();
}

cudaError_t rte_launch_rows(const double* w, void* rows, const int* islot, int N, int nb, int pitch, int Cfull,
                            int fp64, cudaStream_t st) {
  const long long n = (long long)N * nb * Cfull;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (fp64)
    k_rows<double><<<blocks, 256, 0, st>>>(w, static_cast<double*>(rows), islot, N, nb, pitch, Cfull);
  else
    k_rows<float><<<blocks, 256, 0, st>>>(w, static_cast<float*>(rows), islot, N, nb, pitch, Cfull);
  return cudaGetLastError();
}

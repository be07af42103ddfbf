// rte_store.cu -- the pair kernel K(r, r') = exp(-tau(r, r')) dV / (cm |r - r'|^2), tau the path integral of mu_t
// between the voxel centres (FisherInfo_IO/src/kernels.cu:50-148 walks it per pair; rte_walk.cuh does).
//
// The voxels a path crosses and its lengths in them depend on the displacement alone, so a CTA takes all pairs of
// columns at one column displacement (dx, dy), up to `npair` of them, and for every |dz| makes the list of
// (voxel offset, length) once: the crossings of the three axes are arithmetic progressions, so each crossing's
// rank, offset and length follow in closed form and the list is made in parallel.  A pair's integral is then one
// load and one fused multiply-add per voxel crossed, the lanes of a warp taking pairs of the same |dz|.  Lengths
// are integers over Q = 2 max(|dx|,1) max(|dy|,1) max(|dz|,1) and the sum runs in walking order from the
// destination, as path_sum's.  The results of a column pair collect in shared memory and go out as runs of
// destinations per source row; over all sources K is symmetric, so half of the displacements are computed and
// written both ways.  mu_t is read from shared memory (in column order) when it fits, else through L1.
//
// Where voxels couple over a short distance only, displacements of more rows than the column kernels read are left out
// (33^3 L=1 FP64 recomputed, coupling over 2.5 voxels, six terms: all displacements 103 ms, a walk per coupled pair 24,
// now 18).
//
// DERIV: the derivative of K along a direction of mu_t instead, K times minus the path integral of the direction
// (mu: the direction, Kin: K of the same sources, which may be the output).
//
// Bound: instruction issue of the path sums (one add, one load, one multiply-add per voxel crossed) and the barriers
// between lists, sums and write-out.  33^3 FP32: 22.8 ms by a walk per pair (70 % ALU) -> 8.5; FP64 35.3 -> 19;
// 41^3 FP32: 96 -> 46; the sums alone take about half, the write-out a sixth.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "rte_internal.h"
#include "rte_store_plan.h"
#include "rte_walk.cuh"

namespace {

// A voxel of a path: its column offset and z steps from the destination (the sign of z is the pair's), and the
// length in it.  The packed form holds column offsets of grids below 2^21 voxels.
template <typename T, bool PACK>
struct Entry;
template <>
struct __align__(8) Entry<float, true> {
  int code;
  float len;
  __device__ void set(int oc, int oz) { code = oc * 1024 + oz; }
  __device__ int oc() const { return code >> 10; }
  __device__ int oz() const { return code & 1023; }
};
template <>
struct __align__(16) Entry<float, false> {
  int c, z;
  float len, pad;
  __device__ void set(int oc, int oz) { c = oc, z = oz; }
  __device__ int oc() const { return c; }
  __device__ int oz() const { return z; }
};
template <>
struct __align__(16) Entry<double, false> {
  int c, z;
  double len;
  __device__ void set(int oc, int oz) { c = oc, z = oz; }
  __device__ int oc() const { return c; }
  __device__ int oz() const { return z; }
};

static_assert(sizeof(Entry<float, true>) == st_entry_bytes(false, true) &&
                  sizeof(Entry<float, false>) == st_entry_bytes(false, false) &&
                  sizeof(Entry<double, false>) == st_entry_bytes(true, false),
              "list entries as the plan counts them");

template <typename T, bool STAGE, bool PACK, int G, int ST_THREADS, bool DERIV>
__global__ void __launch_bounds__(ST_THREADS, ST_THREADS == 256 ? 3 : (STAGE ? 1 : 2)) k_store_lists(StoreArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x, wid = tid / 32, lane = tid % 32;
  const StLayout Sh(sizeof(T), sizeof(Entry<T, PACK>), a.npair, a.zb, nz, a.cap, STAGE ? a.N : 0);
  Entry<T, PACK>* ent = reinterpret_cast<Entry<T, PACK>*>(smem_raw);
  T* tile = reinterpret_cast<T*>(smem_raw + Sh.off_tile);
  T* lf = reinterpret_cast<T*>(smem_raw + Sh.off_f);       // per |dz|: log2(e) dist / Q (exp2 argument), dV / (cm dist^2)
  size_t* so = reinterpret_cast<size_t*>(smem_raw + Sh.off_o);
  int* ls = reinterpret_cast<int*>(smem_raw + Sh.off_s);   // per |dz|: first entry
  int* cols = reinterpret_cast<int*>(smem_raw + Sh.off_c);  // [npair] destination, [npair] source columns, count
  int& s_unit = cols[2 * a.npair + 1];
  T* smu = reinterpret_cast<T*>(smem_raw + Sh.off_mu);
  constexpr int E = st_pairs_per_lane(sizeof(T) == 8, STAGE);
  const T* gmu = static_cast<const T*>(a.mu);
  if constexpr (STAGE)
    for (int q = tid; q < a.N; q += ST_THREADS) smu[q] = gmu[q];
  const bool whole = a.col0 == 0 && a.col1 == nx * ny;
  const int ry = min(a.ry, ny - 1), noff = whole ? (2 * nx - 1) * ry + nx : (2 * nx - 1) * (2 * ry + 1);
  const int y0 = a.col0 / nx, y1 = (a.col1 - 1) / nx;  // source rows
  const int maxch = (nx * (y1 - y0 + 1) + a.npair - 1) / a.npair, ngrp = (maxch + a.group_ch - 1) / a.group_ch;
  const int zb = a.zb, nblk = (nz + zb - 1) / zb, pitch = zb | 1;
  const T dxf = (T)a.dx, dyf = (T)a.dy, dzf = (T)a.dz, thr = (T)a.prop_thresh;
  // Units (displacement, group of chunks, on few columns also block of z) differ in size: a counter hands them out,
  // group 0 of every displacement first.  Thread 0 draws the next one while the CTA works on this one, past those that
  // do not exist.
  const int nparts = a.zsplit ? nblk * nblk : 1, nunit = noff * ngrp * nparts;
  auto unit = [&](int u, int& dx, int& dy, int& xa, int& wx, int& ya) {  // destination minus source column; its pairs
    const int off = u % noff;
    if (whole) {  // dy = 0, dx >= 0, then dy > 0
      dy = off < nx ? 0 : (off - nx) / (2 * nx - 1) + 1;
      dx = off < nx ? off : (off - nx) % (2 * nx - 1) - (nx - 1);
    } else {
      dy = off / (2 * nx - 1) - ry;
      dx = off % (2 * nx - 1) - (nx - 1);
    }
    xa = max(0, -dx), wx = nx - abs(dx), ya = max(y0, -dy);  // source columns xa.., ya.. of this displacement
    return wx * max(0, min(y1, ny - 1 - max(dy, 0)) - ya + 1);
  };
  auto exists = [&](int u) {
    int q[5];
    return u / noff / nparts * a.group_ch * a.npair < unit(u, q[0], q[1], q[2], q[3], q[4]);
  };
  for (int u = blockIdx.x; u < nunit;) {
    __syncthreads();  // the previous unit's number is read
    if (tid == 0) {
      int n;
      do n = (int)gridDim.x + atomicAdd(a.counter, 1);
      while (n < nunit && !exists(n));
      s_unit = n;
    }
    int dx, dy, xa, wx, ya;
    const int np = unit(u, dx, dy, xa, wx, ya), part = u / noff % nparts, ch0 = u / noff / nparts * a.group_ch;
    const int Dx = abs(dx), Dy = abs(dy), sxy = Dx + Dy;
    const int mx = max(Dx, 1), my = max(Dy, 1);
    const int stx = dx > 0 ? -nz : nz, sty = dy > 0 ? -nx * nz : nx * nz;  // steps towards the source
    // one batch holds all lists of the displacement (ordinary grids): made once for the group's chunks
    const bool once = nblk == 1 && nz * (sxy + 1) + nz * (nz - 1) / 2 <= a.cap;
    for (int ch = ch0; ch < ch0 + a.group_ch && ch * a.npair < np; ++ch)
    for (int bb = part; bb < (a.zsplit ? part + 1 : nblk * nblk); ++bb) {
      // destination z in [d0, d1), source z in [s0, s1)
      const int d0 = bb / nblk * zb, d1 = min(nz, d0 + zb), s0 = bb % nblk * zb, s1 = min(nz, s0 + zb);
      const bool same = whole && dx == 0 && dy == 0;  // a column with itself: blocks below the diagonal by symmetry
      if (same && s0 > d0) continue;
      const int amin = max(0, max(d0 - s1 + 1, s0 - d1 + 1)), amax = max(d1 - 1 - s0, s1 - 1 - d0);
      __syncthreads();  // the previous tile, lists and columns are done with (and mu_t is staged)
      if (wid == 0) {  // the chunk's column pairs, those of the slab's columns
        const int pr = ch * a.npair + lane;
        int cs = -1, cd = 0;
        if (lane < a.npair && pr < np) {
          const int xs = xa + pr % wx, ys = ya + pr / wx;
          cs = ys * nx + xs;
          cd = (ys + dy) * nx + xs + dx;
          if (cs < a.col0 || cs >= a.col1) cs = -1;
        }
        const unsigned m = __ballot_sync(0xffffffffu, cs >= 0);
        if (cs >= 0) {
          const int n = __popc(m & ((1u << lane) - 1));
          cols[n] = cd;
          cols[a.npair + n] = cs;
        }
        if (lane == 0) cols[2 * a.npair] = __popc(m);
      }
      int a0 = amin;
      {  // columns farther apart than voxels couple: zeros, no lists (|dz| only adds to the distance)
        const T hx = (T)Dx * dxf, hy = (T)Dy * dyf, h2 = fma(hx, hx, hy * hy);
        if (h2 > T(0) && !(sqrt(h2) < thr)) {
          for (int e = tid; e < a.npair * zb * pitch; e += ST_THREADS) tile[e] = T(0);
          a0 = amax + 1;
        }
      }
      while (a0 <= amax) {
        int a1 = a0, total = 0;  // lists a0 .. a1 - 1 of this batch
        while (a1 <= amax && total + sxy + a1 + 1 <= a.cap) total += sxy + a1++ + 1;
        if (a0 > amin) __syncthreads();
        if (!once || ch == ch0) {
        for (int da = a0 + ST_THREADS - 1 - tid; da < a1; da += ST_THREADS) {
          const T ex = (T)Dx * dxf, ey = (T)Dy * dyf, ez = (T)da * dzf;
          const T d2 = fma(ex, ex, fma(ey, ey, ez * ez));
          const double x = Dx * a.dx, y = Dy * a.dy, z = da * a.dz, r2 = x * x + y * y + z * z;
          lf[2 * da] = (T)((DERIV ? -1.0 : -1.4426950408889634) * sqrt(r2) / (2.0 * mx * my * max(da, 1)));
          lf[2 * da + 1] = d2 > T(0) && sqrt(d2) < thr ? (T)(a.kscale / r2) : T(0);
        }
        for (int da = a0 + wid; da < a1; da += ST_THREADS / 32) {
          const int first = (da - a0) * (sxy + 1) + (da * (da - 1) - a0 * (a0 - 1)) / 2;
          if (lane == 0) ls[da] = first;
          path_list(Dx, Dy, da, lane, [&](int k, int cx, int cy, int cz, int len, bool) {
            Entry<T, PACK> v;
            v.set(cx * stx + cy * sty, cz);
            v.len = (T)len;
            ent[first + k] = v;
          });
        }
        }
        __syncthreads();
        const int npv = cols[2 * a.npair];
        // lane element: (one of jq pairs) x EE, z, sign of dz; the last chunk of a displacement and grids of few columns
        // have fewer pairs than E
        auto sums = [&](auto ec, int jq) {
          constexpr int EE = decltype(ec)::value;
          for (int ab = a0, rot = wid; ab < a1; ab += 32) {
            // lane l holds list a1 - 1 - (ab - a0) - l, the longest first: the pairs of z at dz = +|dz| and -|dz| and its tasks of 32 elements
            const int da_l = a1 - 1 - (ab - a0) - lane;
            int pl_l = 0, np_l = 0, ml_l = 0, nm_l = 0;
            if (da_l >= a0) {
              pl_l = max(d0, s0 + da_l);
              np_l = max(0, min(d1, s1 + da_l) - pl_l);
              ml_l = max(d0, s0 - da_l);
              nm_l = da_l > 0 ? max(0, min(d1, s1 - da_l) - ml_l) : 0;
            }
            int incl = (jq * (np_l + nm_l) + 31) / 32;
            const int own = incl;
#pragma unroll
            for (int o = 1; o < 32; o *= 2) {
              const int v = __shfl_up_sync(0xffffffffu, incl, o);
              if (lane >= o) incl += v;
            }
            const int ntask = npv > 0 ? __shfl_sync(0xffffffffu, incl, 31) : 0;  // a chunk may miss the slab's columns
            int task = rot;
            for (; task < ntask; task += ST_THREADS / 32) {
              const int l = __ffs(__ballot_sync(0xffffffffu, incl > task)) - 1, da = a1 - 1 - (ab - a0) - l;
              const int f0 = (task - __shfl_sync(0xffffffffu, incl - own, l)) * 32;
              const int pl = __shfl_sync(0xffffffffu, pl_l, l), np_ = __shfl_sync(0xffffffffu, np_l, l);
              const int ml = __shfl_sync(0xffffffffu, ml_l, l), per = np_ + __shfl_sync(0xffffffffu, nm_l, l);
              const bool live = f0 + lane < jq * per;
              const int f = live ? f0 + lane : 0;
              int js = 0, r = f;  // f / per, f % per; js < jq <= 7
              while (r >= per) r -= per, ++js;
              const bool plus = r < np_;
              const int z = plus ? pl + r : ml + r - np_, sg = plus ? -1 : 1;
              uint32_t base[EE];
              T acc[EE];
#pragma unroll
              for (int q = 0; q < EE; ++q) {
                base[q] = (uint32_t)(cols[min(q * jq + js, npv - 1)] * nz + z);
                if constexpr (STAGE) base[q] = (uint32_t)Sh.off_mu + base[q] * (uint32_t)sizeof(T);  // byte offset: one add per load
                acc[q] = T(0);
              }
              const T f1 = lf[2 * da], f2 = lf[2 * da + 1];
              if (f2 != T(0)) {
                const Entry<T, PACK>* le = ent + ls[da];
                const int S = sxy + da;
#pragma unroll (EE < E ? 8 : 2)
                for (int e = 0; e <= S; ++e) {
                  const Entry<T, PACK> v = le[e];
                  const uint32_t at = (uint32_t)(v.oc() + sg * v.oz()) * (STAGE ? (uint32_t)sizeof(T) : 1u);
#pragma unroll
                  for (int q = 0; q < EE; ++q) {
                    T mu;
                    if constexpr (STAGE)
                      mu = *reinterpret_cast<const T*>(smem_raw + (base[q] + at));
                    else
                      mu = __ldg(gmu + (base[q] + at));
                    acc[q] = fma(mu, v.len, acc[q]);
                  }
                }
              }
              if (!live) continue;
              T* to = tile + (js * zb + (z + sg * da - s0)) * pitch + z - d0;  // [pair][source z][destination z]
#pragma unroll
              for (int q = 0; q < EE; ++q) {
                T k;
                if constexpr (DERIV)
                  k = acc[q] * f1;
                else if constexpr (std::is_same<T, float>::value)
                  k = exp2f(acc[q] * f1) * f2;
                else
                  k = exp2(acc[q] * f1) * f2;
                to[q * jq * zb * pitch] = k;
              }
            }
            rot = task - ntask;
          }
        };
        if (npv <= 1)
          sums(std::integral_constant<int, 1>{}, 1);
        else if (npv <= E / 2)
          sums(std::integral_constant<int, E / 2>{}, 1);
        else
          sums(std::integral_constant<int, E>{}, (npv + E - 1) / E);
        a0 = a1;
      }
      __syncthreads();
      // out: the source column's rows, and (all sources) the destination column's rows of the transpose
      T* K = static_cast<T*>(a.K);
      constexpr unsigned KB = 32 * G;
      const unsigned nd = d1 - d0, ns = s1 - s0, md = ((1u << 20) + nd - 1) / nd, ms = ((1u << 20) + ns - 1) / ns;
      const int npv = cols[2 * a.npair], src0 = a.col0 * nz;
      for (unsigned e = tid; e < 2 * npv * (unsigned)zb; e += ST_THREADS) {  // kmat_index(0, position of column and z)
        const unsigned jj = e / zb, zz = e - jj * zb, side = jj >= (unsigned)npv;
        const int col = side ? cols[a.npair + jj - npv] : cols[jj];
        const unsigned p = (unsigned)(col * a.nzp + (side ? s0 : d0)) + zz, o = p % KB;
        size_t& at = so[(side * a.npair + (side ? jj - npv : jj)) * zb + zz];
        if constexpr (DERIV)
          at = (size_t)(p / KB) << 32 | (o % G * 32 + o / G);
        else
          at = (size_t)(p / KB) * a.Kld * KB + o % G * 32 + o / G;
      }
      __syncthreads();
      auto put = [&](size_t at, unsigned src, T v) {  // src: source slot from the slab's first
        if constexpr (DERIV)
          K[((at >> 32) * a.Kld + src) * KB + (uint32_t)at] =
              v * static_cast<const T*>(a.Kin)[((at >> 32) * a.Kin_ld + a.kin_slot + src) * KB + (uint32_t)at];
        else
          K[at + (size_t)src * KB] = v;
      };
      for (unsigned e = tid; e < nd * ns; e += ST_THREADS) {
        const unsigned zs = (e * md) >> 20, zd = e - zs * nd;  // e < 48^2
        for (int j = 0; j < npv; ++j)
          put(so[j * zb + zd], (unsigned)(cols[a.npair + j] * nz + s0 - src0 + (int)zs), tile[(j * zb + zs) * pitch + zd]);
      }
      if (whole)
        for (unsigned e = tid; e < nd * ns; e += ST_THREADS) {
          const unsigned zd = (e * ms) >> 20, zs = e - zd * ns;
          for (int j = 0; j < npv; ++j)
            if (!same || s0 != d0)
              put(so[(a.npair + j) * zb + zs], (unsigned)(cols[j] * nz + d0 + (int)zd), tile[(j * zb + zs) * pitch + zd]);
        }
    }
    __syncthreads();
    u = s_unit;
  }
}

template <typename T, bool STAGE, bool PACK, int G, int ST_THREADS, bool DERIV>
cudaError_t launch_d(StoreArgs a, const StPlan& p, int cap, int sms, cudaStream_t st) {
  void (*kern)(StoreArgs) = k_store_lists<T, STAGE, PACK, G, ST_THREADS, DERIV>;
  a.zb = p.zb;
  a.cap = p.cap;
  a.npair = p.npair;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, ST_THREADS, p.bytes);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  // chunks of column pairs that share one set of lists: as many as leave a few groups for every CTA
  const long long rows = (a.col1 - 1) / a.nx - a.col0 / a.nx + 1, maxch = (a.nx * rows + a.npair - 1) / a.npair;
  const int ry = std::min(a.ry, a.ny - 1);
  const long long noff = a.col0 == 0 && a.col1 == a.nx * a.ny ? (2 * a.nx - 1) * ry + a.nx : (2ll * a.nx - 1) * (2 * ry + 1);
  a.group_ch = (int)std::max<long long>(1, std::min<long long>(8, maxch * noff / (16ll * occ * sms)));
  // few columns, tall ones: the blocks of z are units of their own where the displacements leave CTAs without work
  // (1x1x1000 FP32 1.58 s in seven applications by one CTA)
  a.zsplit = p.zb < a.nz && maxch * noff < 4ll * occ * sms;
  e = cudaMemsetAsync(a.counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<occ * sms, ST_THREADS, p.bytes, st>>>(a);
  return cudaGetLastError();
}

template <typename T, bool STAGE, bool PACK, int G, int ST_THREADS>
cudaError_t launch_t(const StoreArgs& a, const StPlan& p, int cap, int sms, cudaStream_t st) {
  return a.Kin ? launch_d<T, STAGE, PACK, G, ST_THREADS, true>(a, p, cap, sms, st)
               : launch_d<T, STAGE, PACK, G, ST_THREADS, false>(a, p, cap, sms, st);
}

template <typename T, bool STAGE, bool PACK, int G>
cudaError_t launch(const StoreArgs& a, const StPlan& p, int cap, int sms, cudaStream_t st) {
  if constexpr (STAGE)
    if (p.threads == 256) return launch_t<T, STAGE, PACK, G, 256>(a, p, cap, sms, st);
  return launch_t<T, STAGE, PACK, G, 512>(a, p, cap, sms, st);
}

template <int G>
cudaError_t launch_G(const StoreArgs& a, int fp64, int cap, int sms, cudaStream_t st) {
  const StPlan p = st_plan(a.nx, a.ny, a.nz, fp64 != 0, cap);
  if (fp64)
    return p.stage ? launch<double, true, false, G>(a, p, cap, sms, st) : launch<double, false, false, G>(a, p, cap, sms, st);
  if (p.stage) return launch<float, true, true, G>(a, p, cap, sms, st);
  return p.pack ? launch<float, false, true, G>(a, p, cap, sms, st) : launch<float, false, false, G>(a, p, cap, sms, st);
}

}  // namespace

cudaError_t rte_launch_store_kernel(const StoreArgs& a, cudaStream_t st, int fp64) {
  int dev = 0, cap = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (a.group == 3) return launch_G<3>(a, fp64, cap, sms, st);
  if (a.group == 2) return launch_G<2>(a, fp64, cap, sms, st);
  return cudaErrorInvalidValue;
}

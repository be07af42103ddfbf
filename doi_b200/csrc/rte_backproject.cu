// rte_backproject.cu -- symmetric back-projection of the adjoint gradient through exp(-tau).
//
// The path between voxels r and r' is the same set of segments in both directions, so each unordered pair is
// taken once with the weight of both ordered pairs:
//   w(r, r') = k [ (y_r . R(w)) (R(w) . S_r') + (y_r' . P R(w)) (P R(w) . S_r) ],
// w = (r - r') / |r - r'|, P R(w) = R(-w) = (-1)^l R(w).  Pass 1 (k_bp_weights, once per source, summed into Q)
// evaluates the weights, pass 2 (k_bp_walk, once per gradient) adds -w * length to each voxel on the path.
// Both take the pairs of columns at one column displacement (dx, dy) together, dy > 0 or dy = 0, dx >= 0 (the
// destination column's slots follow the source column's).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "rte_device.cuh"
#include "rte_internal.h"
#include "rte_trig.cuh"
#include "rte_walk.cuh"

namespace {

constexpr int BP_THREADS = 256;

// column displacement `off` of (2 nx - 1)(ny - 1) + nx: dy = 0, dx >= 0 first
__device__ __forceinline__ void half_plane(int off, int nx, int& dx, int& dy) {
  dy = off < nx ? 0 : (off - nx) / (2 * nx - 1) + 1;
  dx = off < nx ? off : (off - nx) % (2 * nx - 1) - (nx - 1);
}

// the column pairs of chunk `ch` (npair a chunk) at (dx, dy): [0, npair) destination, [npair, 2 npair) source
// columns; returns how many there are
__device__ __forceinline__ int chunk_columns(int ch, int npair, int np, int nx, int dx, int dy, int* cols) {
  const int wx = nx - abs(dx), xa = max(0, -dx), n = min(npair, np - ch * npair);
  for (int q = threadIdx.x; q < n; q += BP_THREADS) {
    const int pr = ch * npair + q, xs = xa + pr % wx, ys = pr / wx;
    cols[q] = (ys + dy) * nx + xs + dx;
    cols[npair + q] = ys * nx + xs;
  }
  return n;
}

// -------------------------------------------------------------------------------------------------
// Pass 1.  On the meridian of a column pair a row of coefficients contracts to 2L+1 numbers (rte_trig.cuh), y and
// S of both columns once per pair of columns, so a pair of voxels costs four dot products of 2L+1 instead of four
// of (L+1)^2 and an SH recurrence.  The trigonometric values of the displacements are FP64 values rounded to T.
// A thread keeps the two contracted rows of one destination and goes through the sources of its column, whose rows
// every lane reads (broadcast).  Bound by the latency of the loads of K and Q and of the contracted rows' making
// (issue 42 %, shared memory 58 %).  33^3 L=5, per source: 17.8 ms by spherical harmonics per pair on 64 x 64 tiles
// -> 9.3.
template <int L>
__host__ __device__ constexpr int bw_row() {
  return 2 * L + 2;  // (cos k, sin k) k = 1..L, then (k = 0, 0)
}

// two contracted rows of one voxel, an odd number of 16-byte units apart
template <int L, typename T>
__host__ __device__ constexpr int bw_pitch() {
  const int unit = 16 / (int)sizeof(T), n = (2 * bw_row<L>() + unit - 1) / unit;
  return (n | 1) * unit;
}

template <int L, typename T>
struct BwLayout {  // rows [npair][source, destination][zb] | trigonometric pairs [L][2 zb] | azimuth | columns
  size_t off_t, off_a, off_c, bytes;
  __host__ __device__ BwLayout(int npair, int zb) {
    off_t = sizeof(T) * 2 * npair * zb * bw_pitch<L, T>();
    off_a = off_t + sizeof(T) * 2 * L * 2 * zb;
    off_c = off_a + sizeof(T) * (2 * L + 2);
    bytes = off_c + sizeof(int) * 2 * npair;
  }
};

template <int L, typename T>
__global__ void __launch_bounds__(BP_THREADS, sizeof(T) == 4 ? (L <= 5 ? 3 : 2) : (L <= 4 ? 2 : 1)) k_bp_weights(BpArgs a) {
  constexpr int C = (L + 1) * (L + 1), NT = bw_row<L>(), RP = bw_pitch<L, T>();
  constexpr bool F32 = std::is_same<T, float>::value;
  typedef typename std::conditional<F32, float2, double2>::type T2;
  typedef typename std::conditional<F32, float4, double2>::type Vec;
  constexpr int VN = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x, wid = tid / 32, lane = tid % 32, npair = a.jq, zb = a.zb;
  const BwLayout<L, T> Sh(npair, zb);
  T* sB = reinterpret_cast<T*>(smem_raw);
  T2* sT = reinterpret_cast<T2*>(smem_raw + Sh.off_t);
  T* sA = reinterpret_cast<T*>(smem_raw + Sh.off_a);
  int* cols = reinterpret_cast<int*>(smem_raw + Sh.off_c);
  const int noff = (2 * nx - 1) * (ny - 1) + nx, nblk = (nz + zb - 1) / zb;
  const int ngrp = ((nx * ny + npair - 1) / npair + a.group_ch - 1) / a.group_ch;
  const T* rows[2] = {static_cast<const T*>(a.S), static_cast<const T*>(a.y)};
  T* Q = static_cast<T*>(a.Q);
  const int kb = 32 * a.group;
  for (long long w = blockIdx.x; w < (long long)noff * ngrp * a.nparts; w += gridDim.x) {
    int dx, dy;
    half_plane((int)(w % noff), nx, dx, dy);
    const int part = (int)(w / noff % a.nparts), ch0 = (int)(w / noff / a.nparts) * a.group_ch;
    const int np = (nx - abs(dx)) * (ny - dy);
    if (ch0 * npair >= np) continue;
    const bool same = dx == 0 && dy == 0;
    const double ex = dx * a.dx, ey = dy * a.dy, rho = sqrt(ex * ex + ey * ey);
    const bool far = rho >= a.prop_thresh;  // no coupling, and the stored kernel may not hold these pairs
    for (int bb = part; bb < nblk * nblk; bb += a.nparts) {
      const int d0 = bb / nblk * zb, d1 = min(nz, d0 + zb), s0 = bb % nblk * zb, s1 = min(nz, s0 + zb);
      const int nd = d1 - d0, ns = s1 - s0, e0 = d0 - s1 + 1;  // displacements e0 .. d1 - 1 - s0
      if (same && s0 >= d1) continue;
      for (int ch = ch0; ch < ch0 + a.group_ch && ch * npair < np; ++ch) {
        __syncthreads();  // the previous chunk's rows and columns are done with
        const int npv = chunk_columns(ch, npair, np, nx, dx, dy, cols);
        if (ch == ch0) {
          for (int e = tid; e < nd + ns - 1; e += BP_THREADS) {
            const double ez = (e0 + e) * a.dz, r = sqrt(rho * rho + ez * ez);
            const double ct = r > 0.0 ? ez / r : 1.0, st = r > 0.0 ? rho / r : 0.0;
            double c = 1.0, s = 0.0;
#pragma unroll
            for (int k = 0; k < L; ++k) {
              const double n = c * ct - s * st;
              s = c * st + s * ct;
              c = n;
              T2 v;
              v.x = (T)c;
              v.y = (T)s;
              sT[k * 2 * zb + e] = v;
            }
          }
          if (tid == 0) {
            const double cp = rho > 0.0 ? ex / rho : 1.0, sp = rho > 0.0 ? ey / rho : 0.0;
            double c = 1.0, s = 0.0;
            for (int m = 1; m <= L; ++m) {
              const double n = c * cp - s * sp;
              s = c * sp + s * cp;
              c = n;
              sA[2 * m - 2] = (T)c;
              sA[2 * m - 1] = (T)s;
            }
          }
        }
        __syncthreads();
        // contract: voxel q of a column pair (sources, then destinations), first S (o = 0), then y; the row that
        // meets P R gets its odd orders negated.  Source: (S, P y), destination: (y, P S).
        for (int e = tid; e < npv * (ns + nd) * 2; e += BP_THREADS) {
          const int o = e & 1, f = e >> 1, p = f / (ns + nd), q = f - p * (ns + nd), side = q >= ns;
          const int z = side ? d0 + q - ns : s0 + q, col = cols[side ? p : npair + p];
          const T* src = rows[o] + ((size_t)col * nz + z) * a.pitch;
          const bool par = side != o;  // source y, destination S
          T row[C];
#pragma unroll
          for (int c = 0; c < C; c += VN) {
            const Vec v = *reinterpret_cast<const Vec*>(src + c);
            row[c] = v.x;
            if (c + 1 < C) row[c + 1] = v.y;
            if constexpr (F32) {
              if (c + 2 < C) row[c + 2] = v.z;
              if (c + 3 < C) row[c + 3] = v.w;
            }
          }
          if (par) {
#pragma unroll
            for (int l = 1; l <= L; l += 2)
#pragma unroll
              for (int c = l * l; c < (l + 1) * (l + 1); ++c) row[c] = -row[c];
          }
          T b[nb_row<L>()];
          contract_row<L, T>(row, sA, b);
          T* d = sB + ((p * 2 + side) * zb + (z - (side ? d0 : s0))) * RP + (par ? NT : 0);
#pragma unroll
          for (int k = 0; k < NT; ++k) d[k] = b[k];
        }
        __syncthreads();
        const int nel = (npv * nd + 31) / 32, seg = (ns + 3) / 4;
        for (int task = wid; task < nel * 4; task += BP_THREADS / 32) {
          const int f = task / 4 * 32 + lane, zs0 = task % 4 * seg, zs1 = min(ns, zs0 + seg);
          const bool live = f < npv * nd;
          const int p = live ? f / nd : 0, zd = live ? f - p * nd : 0;
          const int cd = cols[p], cs = cols[npair + p], d = cd * nz + d0 + zd, sl0 = cs * nz + s0;
          T yd[NT], sd[NT];
          {
            const T* v = sB + ((p * 2 + 1) * zb + zd) * RP;
#pragma unroll
            for (int k = 0; k < NT; ++k) yd[k] = v[k], sd[k] = v[NT + k];
          }
          const T* B = sB + (p * 2) * zb * RP;
          const int pos = kmat_pos(d, nz, a.nzp);
          const size_t k0 = (size_t)(pos / kb) * a.Kld * kb + pos % kb % a.group * 32 + pos % kb / a.group;
          T* q = Q + (size_t)sl0 * a.ld + d;
#pragma unroll 2
          for (int zs = zs0; zs < zs1; ++zs) {
            const bool on = live && !(same && s0 + zs >= d0 + zd);
            T kk = T(0), old = T(0);
            if (on) {
              if (a.accumulate) old = q[(size_t)zs * a.ld];
              if (far)
                kk = T(0);
              else if (a.Kmat64)
                kk = (T)__ldg(a.Kmat64 + k0 + (size_t)(sl0 + zs) * kb);
              else if (a.Kmat)
                kk = (T)__ldg(a.Kmat + k0 + (size_t)(sl0 + zs) * kb);
              else {
                const T fx = (T)dx * (T)a.dx, fy = (T)dy * (T)a.dy, fz = (T)(d0 + zd - s0 - zs) * (T)a.dz;
                const T d2 = fx * fx + fy * fy + fz * fz, dist = sqrt(d2);
                if (dist < (T)a.prop_thresh) {
                  int Q0;
                  const T ps = path_sum<T, double>(cd / nx, cd % nx, d0 + zd, cs / nx, cs % nx, s0 + zs, a.mut, nz,
                                                   nx * nz, Q0);
                  kk = exp(-ps * dist / (T)Q0) * (T)a.kscale / d2;
                }
              }
            }
            const T* v = B + zs * RP;
            const T2* tr = sT + (d0 + zd) - (s0 + zs) - e0;
            T wt;
            if constexpr (F32) {
              f2_t vs[NT], ac[4];
#pragma unroll
              for (int c = 0; c < NT / 2; ++c) {
                const ulonglong2 x = reinterpret_cast<const ulonglong2*>(v)[c];
                vs[2 * c] = x.x;
                vs[2 * c + 1] = x.y;
              }
              ac[0] = f2_pack(yd[2 * L], 0.f);
              ac[1] = vs[L];
              ac[2] = vs[2 * L + 1];
              ac[3] = f2_pack(sd[2 * L], 0.f);
#pragma unroll
              for (int k = 0; k < L; ++k) {
                const f2_t t = *reinterpret_cast<const f2_t*>(tr + k * 2 * zb);
                ac[0] = f2_fma(t, f2_pack(yd[2 * k], yd[2 * k + 1]), ac[0]);
                ac[1] = f2_fma(t, vs[k], ac[1]);
                ac[2] = f2_fma(t, vs[L + 1 + k], ac[2]);
                ac[3] = f2_fma(t, f2_pack(sd[2 * k], sd[2 * k + 1]), ac[3]);
              }
              float x[4], lo, hi;
#pragma unroll
              for (int i = 0; i < 4; ++i) f2_unpack(ac[i], lo, hi), x[i] = lo + hi;
              wt = kk * fma(x[0], x[1], x[2] * x[3]);
            } else {
              T a1 = yd[2 * L], b1 = v[2 * L], a2 = v[NT + 2 * L], b2 = sd[2 * L];
#pragma unroll
              for (int k = 0; k < L; ++k) {
                const T2 t = tr[k * 2 * zb];
                a1 = fma(t.x, yd[2 * k], fma(t.y, yd[2 * k + 1], a1));
                b1 = fma(t.x, v[2 * k], fma(t.y, v[2 * k + 1], b1));
                a2 = fma(t.x, v[NT + 2 * k], fma(t.y, v[NT + 2 * k + 1], a2));
                b2 = fma(t.x, sd[2 * k], fma(t.y, sd[2 * k + 1], b2));
              }
              wt = kk * fma(a1, b1, a2 * b2);
            }
            if (on) q[(size_t)zs * a.ld] = old + wt;
          }
        }
      }
    }
  }
}

// -------------------------------------------------------------------------------------------------
// Pass 2, the transpose of the path integrals of rte_store.cu.  At one column displacement a path of |dz| visits
// the same column steps j for every pair of columns, and in step j the entries [jst(|dz|, j), jst(|dz|, j + 1)) of
// the list of |dz|.  So a lane takes voxel z of step j of E column pairs and gathers, over every |dz| and entry,
// the weights of the pairs whose path has that entry there:
//   dest above the source: row (+, |dz|) at u = z + cz - |dz|,  below: row (-, |dz|) at u = z - cz,
// u the lower end's z.  The rows of weights lie in shared memory one after another, each with |dz| + 1 or more zeros
// behind its nz - |dz| values, so that entries whose pair does not exist read zeros: no test per entry, one list
// entry read for 2 E weights, and no atomics but one FP64 addition per lane, pair and step (atomics on a shared
// copy of the gradient per voxel crossed in their place: 86.7 ms at 33^3, now 29.1).  Where the columns are too long for
// one batch of lists and rows, a batch of |dz| is a unit of work of its own.
constexpr int BP_E = 3;
constexpr int BP_CAP = 3072;  // most list entries of a batch (one list has at most 3 * 1023 + 1)

template <typename T>
struct __align__(2 * sizeof(T)) BpEntry {
  T len;
  int z;
};

// entries [cap] | zeros [pitch], rows [pairs][2][rows][pitch] | step starts [2 cap] | column steps [nx + ny], columns
template <typename T>
struct WalkLayout {
  size_t off_t, off_j, off_o, off_c, bytes;
  __host__ __device__ WalkLayout(int npair, int rows, int nz, int cap, int nxy) {
    off_t = sizeof(BpEntry<T>) * cap;
    off_j = off_t + sizeof(T) * ((size_t)2 * npair * rows + 1) * ((nz + 1) | 1);
    off_o = (off_j + sizeof(uint16_t) * 2 * cap + 3) / 4 * 4;
    off_c = off_o + sizeof(int) * nxy;
    bytes = off_c + sizeof(int) * 2 * npair;
  }
};

template <typename T>
__global__ void __launch_bounds__(BP_THREADS) k_bp_walk(BpArgs a) {
  constexpr int E = BP_E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x, wid = tid / 32, lane = tid % 32;
  const int jq = a.jq, npair = E * jq, pitch = (nz + 1) | 1, rows = a.rows;
  const WalkLayout<T> Sh(npair, rows, nz, a.cap, nx + ny);
  BpEntry<T>* ent = reinterpret_cast<BpEntry<T>*>(smem_raw);
  T* tile = reinterpret_cast<T*>(smem_raw + Sh.off_t);
  uint16_t* jst = reinterpret_cast<uint16_t*>(smem_raw + Sh.off_j);
  int* oc = reinterpret_cast<int*>(smem_raw + Sh.off_o);
  int* cols = reinterpret_cast<int*>(smem_raw + Sh.off_c);
  const int noff = (2 * nx - 1) * (ny - 1) + nx, ntile = (2 * npair * rows + 1) * pitch;
  const int ngrp = ((nx * ny + npair - 1) / npair + a.group_ch - 1) / a.group_ch;
  const T* Q = static_cast<const T*>(a.Q);
  for (int e = tid; e < ntile; e += BP_THREADS) tile[e] = T(0);
  int rot = wid;
  for (long long w = blockIdx.x; w < (long long)noff * ngrp * a.nparts; w += gridDim.x) {
    int dx, dy;
    half_plane((int)(w % noff), nx, dx, dy);
    const int part = (int)(w / noff % a.nparts), ch0 = (int)(w / noff / a.nparts) * a.group_ch;
    const int np = (nx - abs(dx)) * (ny - dy);
    if (ch0 * npair >= np) continue;
    const bool same = dx == 0 && dy == 0;
    const int A1 = a.single ? nz : min(nz, (part + 1) * rows);  // this unit's |dz|: all, or one batch of rows
    const int Dx = abs(dx), Dy = dy, sxy = Dx + Dy, stx = dx > 0 ? -1 : 1, sty = -nx;  // steps towards the source
    for (int ch = ch0; ch < ch0 + a.group_ch && ch * npair < np; ++ch)
      for (int a0 = a.single ? 0 : part * rows; a0 < A1;) {
        int a1 = a0, total = 0;  // lists a0 .. a1 - 1 of this batch
        while (a1 < A1 && total + sxy + a1 + 1 <= a.cap) total += sxy + a1++ + 1;
        __syncthreads();  // the previous batch's rows, lists and columns are done with
        const int npv = chunk_columns(ch, npair, np, nx, dx, dy, cols);
        if (!a.single || ch == ch0)
          for (int da = a0 + wid; da < a1; da += BP_THREADS / 32) {
            const int first = (da - a0) * (sxy + 1) + (da * (da - 1) - a0 * (a0 - 1)) / 2;
            const int jf = (da - a0) * (sxy + 2);
            const double ex = Dx * a.dx, ey = Dy * a.dy, ez = da * a.dz;
            const T coef = (T)(-sqrt(ex * ex + ey * ey + ez * ez) / (2.0 * max(Dx, 1) * max(Dy, 1) * max(da, 1)));
            if (lane == 0) {
              jst[jf] = (uint16_t)first;
              jst[jf + sxy + 1] = (uint16_t)(first + sxy + da + 1);
            }
            path_list(Dx, Dy, da, lane, [&](int k, int cx, int cy, int cz, int len, bool leaves) {
              BpEntry<T> v;
              v.len = coef * (T)len;
              v.z = cz;
              ent[first + k] = v;
              if (leaves) jst[jf + cx + cy + 1] = (uint16_t)(first + k + 1);
              if (da == a0) oc[cx + cy] = cx * stx + cy * sty;
            });
          }
        if (!a.single) {  // another batch's rows: their zeros lie elsewhere
          for (int e = tid; e < ntile; e += BP_THREADS) tile[e] = T(0);
        }
        __syncthreads();
        // a single batch: the pairs of a column pair in the order they lie in; else only those of the batch
        const int nel = a.single ? nz * nz : 2 * nz * (a1 - a0);
        for (int e = tid; e < nel; e += BP_THREADS) {
          int zs = e / nz, zd = e - zs * nz;
          if (!a.single) {
            const int d = a0 + zs / 2, up = zs & 1, u = zd;
            if (u + d >= nz || (up && d == 0)) continue;
            zs = up ? u + d : u, zd = up ? u : u + d;
          }
          const int da = abs(zd - zs);
          T* to = tile + pitch + ((zd < zs ? rows : 0) + da - a0) * pitch + min(zs, zd);
          const bool on = !same || zs < zd;
          for (int p = 0; p < npv; ++p)
            to[2 * p * rows * pitch] =
                on ? Q[(size_t)(cols[npair + p] * nz + zs) * a.ld + cols[p] * nz + zd] : T(0);
        }
        __syncthreads();
        const int nbk = (jq * nz + 31) / 32, ntask = (sxy + 1) * nbk;
        int task = rot;
        for (; task < ntask; task += BP_THREADS / 32) {
          const int j = task / nbk, f = (task - j * nbk) * 32 + lane;
          const bool live = f < jq * nz;
          const int js = live ? f / nz : 0, z = live ? f - js * nz : 0;
          const T* base = tile + pitch + js * 2 * rows * pitch + z;
          const int qs = jq * 2 * rows * pitch, ms = rows * pitch;
          T acc[E];
#pragma unroll
          for (int q = 0; q < E; ++q) acc[q] = T(0);
          for (int da = a0; da < a1; ++da) {
            const uint16_t* js_ = jst + (da - a0) * (sxy + 2) + j;
            const int e1 = js_[1];
            const T* rp = base + (da - a0) * pitch - da;
            const T* rm = base + (da - a0) * pitch + ms;
#pragma unroll 2
            for (int e = js_[0]; e < e1; ++e) {
              const BpEntry<T> v = ent[e];
              const T* pp = rp + v.z;
              const T* pm = rm - v.z;
#pragma unroll
              for (int q = 0; q < E; ++q) acc[q] = fma(v.len, pp[q * qs], acc[q]);
#pragma unroll
              for (int q = 0; q < E; ++q) acc[q] = fma(v.len, pm[q * qs], acc[q]);
            }
          }
#pragma unroll
          for (int q = 0; q < E; ++q)
            if (live && q * jq + js < npv) atomicAdd(a.gcol + (size_t)(cols[q * jq + js] + oc[j]) * nz + z, (double)acc[q]);
        }
        rot = task - ntask;
        a0 = a1;
      }
  }
}

__global__ void k_bp_add(const double* gcol, const int* islot, double* g, int N) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < N) g[r] += gcol[islot[r]];
}

struct Device {
  int cap = 0, sms = 0;
  cudaError_t err;
  Device() {
    int dev = 0;
    err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
};

// one wave of CTAs over the (displacement, group of chunks) units, chunks per group as many as leave several
// groups for every CTA
// nparts: into how many parts a unit's |dz| or blocks of z can be divided; `split` does it only where the units leave
// CTAs without work (few columns, tall ones: the weights of 1x1x600 by one CTA)
cudaError_t launch_units(void (*kern)(BpArgs), BpArgs a, int npair, size_t smem, int nparts, bool split, const Device& d,
                         cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, d.cap);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BP_THREADS, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  const long long maxch = ((long long)a.nx * a.ny + npair - 1) / npair, noff = (2ll * a.nx - 1) * (a.ny - 1) + a.nx;
  a.group_ch = (int)std::max<long long>(1, std::min<long long>(8, maxch * noff / (16ll * occ * d.sms)));
  a.nparts = split && maxch * noff >= 4ll * occ * d.sms ? 1 : nparts;
  const long long units = noff * ((maxch + a.group_ch - 1) / a.group_ch) * a.nparts;
  kern<<<(unsigned)std::min<long long>(units, (long long)occ * d.sms), BP_THREADS, smem, st>>>(a);
  return cudaGetLastError();
}

template <int L, typename T>
cudaError_t launch_weights(BpArgs a, cudaStream_t st) {
  const Device d;
  if (d.err != cudaSuccess) return d.err;
  const int nblk = (a.nz + 47) / 48;
  a.zb = (a.nz + nblk - 1) / nblk;
  // column pairs per chunk: up to 256 destinations, two or three CTAs per SM
  a.jq = 1;
  while (a.jq * a.zb < 256 && BwLayout<L, T>(a.jq + 1, a.zb).bytes <= 72 * 1024) ++a.jq;
  return launch_units(k_bp_weights<L, T>, a, a.jq, BwLayout<L, T>(a.jq, a.zb).bytes, nblk * nblk, true, d, st);
}

template <int L>
cudaError_t launch_weights_L(const BpArgs& a, int fp64, cudaStream_t st) {
  return fp64 ? launch_weights<L, double>(a, st) : launch_weights<L, float>(a, st);
}

template <typename T>
cudaError_t launch_walk(BpArgs a, cudaStream_t st) {
  const Device d;
  if (d.err != cudaSuccess) return d.err;
  cudaError_t e = cudaMemsetAsync(a.gcol, 0, sizeof(double) * a.N, st);
  if (e != cudaSuccess) return e;
  const int nxy = a.nx + a.ny, longest = nxy - 1 + a.nz;
  const long long all = (long long)a.nz * (nxy - 1) + (long long)a.nz * (a.nz - 1) / 2;  // lists of the longest displacement
  a.cap = (int)std::min<long long>(std::max(longest, BP_CAP), all);
  a.cap = (std::max(a.cap, longest) + 1) / 2 * 2;
  // lanes of a step: jq * nz; of the jq whose rows fit two CTAs per SM, the one that leaves fewest lanes idle
  const size_t budget = 110 * 1024;
  a.jq = 1;
  a.rows = a.nz;
  double best = 0.0;
  for (int jq = 1; jq <= 8 && WalkLayout<T>(BP_E * jq, a.nz, a.nz, a.cap, nxy).bytes <= budget; ++jq) {
    const int lanes = jq * a.nz;
    const double eff = (double)lanes / ((lanes + 31) / 32 * 32);
    if (eff > best + 0.02) best = eff, a.jq = jq;
  }
  while (a.rows > 1 && WalkLayout<T>(BP_E * a.jq, a.rows, a.nz, a.cap, nxy).bytes > budget) --a.rows;
  const size_t smem = WalkLayout<T>(BP_E * a.jq, a.rows, a.nz, a.cap, nxy).bytes;
  if (smem > (size_t)d.cap) return cudaErrorInvalidValue;
  a.single = a.rows == a.nz && all <= a.cap;
  e = launch_units(k_bp_walk<T>, a, BP_E * a.jq, smem, a.single ? 1 : (a.nz + a.rows - 1) / a.rows, false, d, st);
  if (e != cudaSuccess) return e;
  k_bp_add<<<(a.N + 255) / 256, 256, 0, st>>>(a.gcol, a.islot, a.g, a.N);
  return cudaGetLastError();
}

}  // namespace

cudaError_t rte_launch_bp_weights(const BpArgs& a, int LA, int fp64, cudaStream_t st) {
  switch (LA) {
    case 0: return launch_weights_L<0>(a, fp64, st);
    case 1: return launch_weights_L<1>(a, fp64, st);
    case 2: return launch_weights_L<2>(a, fp64, st);
    case 3: return launch_weights_L<3>(a, fp64, st);
    case 4: return launch_weights_L<4>(a, fp64, st);
    case 5: return launch_weights_L<5>(a, fp64, st);
    case 6: return launch_weights_L<6>(a, fp64, st);
    case 7: return launch_weights_L<7>(a, fp64, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t rte_launch_bp_walk(const BpArgs& a, int fp64, cudaStream_t st) {
  return fp64 ? launch_walk<double>(a, st) : launch_walk<float>(a, st);
}

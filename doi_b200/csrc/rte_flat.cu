// rte_flat.cu -- flat grids: columns along x or y in place of z.
//
// The column form (rte_column.cu, rte_store.cu, rte_backproject.cu) pays the contraction of a source row and the
// expansion of a destination's sums once per pair of columns, so columns of a few voxels leave it nothing to share:
// 110x110x1 L=3, mixed, kernel stored, six terms and the final application 197 ms, recomputed 910 (by a walk and
// spherical harmonics per pair 10.3 and 104).  The operator commutes with exchanging axes, A P = P A, P acting on a
// distribution by the voxel order and, within each degree, by an orthogonal matrix M on the coefficients.  A flat grid
// is therefore solved in the frame whose column axis is its longest one: the rows of the pair kernels are M w
// (k_rows_rot), the chunk sums come back by the transpose of M (k_sums_rot), and all else stays as it is.
// 110x110x1 L=3 so: 5.0 and 16.7 ms.
//
// The reference's snapped direction table (FisherInfo_IO/src/kernels.cu:326-333) does not commute with it: its cells
// lie about the z axis.  Flat grids of that model keep the pair kernel in the exchanged frame, which is a scalar per
// pair, and apply it pair by pair with the snapped direction of each displacement from a table (k_pair_dirs).
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "rte_device.cuh"
#include "rte_internal.h"

namespace {

// voxel-order rows [N][nb][Cfull] -> column-order rows [nb][N][pitch] of M w, coefficient c times N_c
template <typename T>
__global__ void k_rows_rot(const double* w, T* rows, const double* M, const int* islot, int N, int nb, int pitch, int Cfull) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int vstride = nb * Cfull;
  if (t >= (long long)N * vstride) return;
  const int r = (int)(t / vstride), e = (int)(t % vstride);
  const int rhs = e / Cfull, c = e - rhs * Cfull;
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  const double* x = w + t - c;
  double v = 0.0;
  for (int q = l * l; q < (l + 1) * (l + 1); ++q) v = fma(__ldg(M + c * Cfull + q), __ldg(x + q), v);
  rows[((size_t)rhs * N + islot[r]) * pitch + c] = (T)(v * kMonic.N[c]);
}

// chunk sums of the exchanged frame's voxels -> FP64 sums [N][nb][Cfull] of the grid's, by the transpose of M (null: as
// they are).  A thread adds the chunks of one element, a block of whole rows exchanges them through shared memory.
template <typename T>
__global__ void k_sums_rot(FlatArgs a, int Cact) {
  __shared__ double sh[256];
  const int per = blockDim.x / a.Cfull, vstride = a.nb * a.Cfull;  // rows (voxel, right-hand side) of a block
  const long long row = (long long)blockIdx.x * per + threadIdx.x / a.Cfull;
  const int c = threadIdx.x % a.Cfull, r = (int)(row / a.nb), rhs = (int)(row - (long long)r * a.nb);
  const bool act = r < a.N && c < Cact;
  double v = 0.0;
  if (act) {
    const int x = r % a.nx, y = r / a.nx % a.ny, z = r / (a.nx * a.ny);
    const T* p = static_cast<const T*>(a.part) + (size_t)(x * a.sx + y * a.sy + z * a.sz) * vstride + rhs * a.Cfull + c;
    const size_t ld = (size_t)a.N * vstride;
#pragma unroll 8
    for (int s = 0; s < a.S; ++s) v += (double)p[s * ld];
    if (std::is_same<T, float>::value) v *= kMonic.N[c];
  }
  if (a.M) {
    sh[threadIdx.x] = v;
    __syncthreads();
    int l = 0;
    while ((l + 1) * (l + 1) <= c) ++l;
    v = 0.0;
    for (int q = l * l; q < (l + 1) * (l + 1); ++q) v = fma(__ldg(a.M + q * a.Cfull + c), sh[threadIdx.x - c + q], v);
  }
  if (act) a.out[(size_t)row * a.Cfull + c] = v;
}

// Snapped directions of the displacements destination minus source (transposed: source minus destination), x fastest.
template <typename V, typename T>
__global__ void k_dirs_table(int nx, int ny, int nz, double dx, double dy, double dz, int transpose, V* tab) {
  const int mx = 2 * nx - 1, my = 2 * ny - 1, mz = 2 * nz - 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= mx * my * mz) return;
  const int sg = transpose ? -1 : 1;
  const double fx = (double)(sg * (t % mx - (nx - 1))) * dx, fy = (double)(sg * (t / mx % my - (ny - 1))) * dy,
               fz = (double)(sg * (t / (mx * my) - (nz - 1))) * dz;
  const double dist = sqrt(fx * fx + fy * fy + fz * fz);
  double ux = 0.0, uy = 0.0, uz = 1.0;
  if (dist > 0.0) table_direction(fx, fy, fz, dist, ux, uy, uz);
  V v;
  v.x = (T)ux;
  v.y = (T)uy;
  v.z = (T)uz;
  v.w = T(0);
  tab[t] = v;
}

constexpr int PD_CTA = 128, PD_TS = 32;  // destinations of a CTA, sources staged at a time

// The pair kernel applied pair by pair: one thread per destination (the lanes of a warp those whose kernel values lie
// side by side), sources in runs of PD_TS through shared memory.  Monic spherical harmonics U (kMonic): the rows hold
// N_c W_c.  FP32 at L >= 7 evaluates them in FP64, as the column kernels tabulate them there.  Bound by instruction
// issue (5 C multiply-adds and a 16-byte direction a pair).  100x100x1 L=2,
// six terms and the final application, mixed, kernel stored: 126 ms on z columns, 6.2 here (26 by a direction computed per
// pair).
template <int L, typename T>
__global__ void __launch_bounds__(PD_CTA) k_pair_dirs(ColArgs a) {
  constexpr int C = (L + 1) * (L + 1);
  typedef typename std::conditional<std::is_same<T, double>::value || L >= 7, double, float>::type D;
  typedef typename std::conditional<std::is_same<D, double>::value, double4, float4>::type V;
  __shared__ T sW[PD_TS * C];
  __shared__ int sd[PD_TS];
  const int tid = threadIdx.x, lane = tid % 32, wi = blockIdx.x * (PD_CTA / 32) + tid / 32, kb = 32 * a.group;
  const int blk = wi / a.group, i = wi % a.group, p = blk * kb + lane * a.group + i;
  const int col = p / a.nzp, z = p - col * a.nzp, ncol = a.nx * a.ny;
  const bool act = col < ncol && z < a.nz;
  const int bd = a.d0 + z * a.dsz + col % a.nx * a.dsx + col / a.nx * a.dsy;  // entry of displacement 0 from here
  const int rhs = blockIdx.z;
  const T* W = static_cast<const T*>(a.W) + (size_t)rhs * a.N * a.pitch;
  const T* K = static_cast<const T*>(a.K) + (size_t)blk * a.Kld * kb + i * 32 + lane;
  const V* dirs = static_cast<const V*>(a.tab);
  if (blockIdx.x == 0 && blockIdx.y == 0 && rhs == 0 && tid < 4 && a.red) a.red[tid] = 0.0;
  // sources of this chunk in the rows that the CTA's destinations can couple with (others' kernel values are not written)
  const int w0 = blockIdx.x * (PD_CTA / 32), c0 = w0 / a.group * kb / a.nzp;
  const int c1 = (((w0 + PD_CTA / 32 - 1) / a.group + 1) * kb - 1) / a.nzp;
  const int s_beg = max(a.col0 + (int)blockIdx.y * a.chunk, (c0 / a.nx - a.ry) * a.nx) * a.nz;
  const int s_end = min(min(a.col1, a.col0 + ((int)blockIdx.y + 1) * a.chunk), (c1 / a.nx + a.ry + 1) * a.nx) * a.nz;
  T acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = T(0);
  for (int s0 = s_beg; s0 < s_end; s0 += PD_TS) {
    const int ns = min(PD_TS, s_end - s0);
    __syncthreads();
    for (int q = tid; q < ns * C; q += PD_CTA) sW[q] = W[(size_t)(s0 + q / C) * a.pitch + q % C];
    for (int q = tid; q < ns; q += PD_CTA) {
      const int sc = (s0 + q) / a.nz, sz = (s0 + q) % a.nz;
      sd[q] = sz * a.dsz + sc % a.nx * a.dsx + sc / a.nx * a.dsy;
    }
    __syncthreads();
    if (!act) continue;
    for (int q = 0; q < ns; ++q) {
      const T kk = K[(size_t)(s0 + q - a.kslot0) * kb];
      if (kk == T(0)) continue;
      const V u = dirs[bd - sd[q]];
      T U[C];
      {
        D cm = D(1), sm = D(0);
#pragma unroll
        for (int m = 0; m <= L; ++m) {
          if (m > 0) {
            const D n = m == 1 ? (D)u.x : cm * (D)u.x - sm * (D)u.y;
            sm = m == 1 ? (D)u.y : cm * (D)u.y + sm * (D)u.x;
            cm = n;
          }
          D c1 = cm, s1 = sm, c0 = D(0), s0_ = D(0);
#pragma unroll
          for (int l = m; l <= L; ++l) {
            if (l > m) {
              const D b = l > m + 1 ? (D)kMonic.beta[l * (l + 1) / 2 + m] : D(0);
              const D cn = fma((D)u.z, c1, -b * c0), sn = fma((D)u.z, s1, -b * s0_);
              c0 = c1, c1 = cn, s0_ = s1, s1 = sn;
            }
            U[l * l + l + m] = (T)c1;
            if (m > 0) U[l * l + l - m] = (T)s1;
          }
        }
      }
      const T* w = sW + q * C;
      T S = T(0);
#pragma unroll
      for (int c = 0; c < C; ++c) S = fma(U[c], w[c], S);
      S *= kk;
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = fma(U[c], S, acc[c]);
    }
  }
  if (!act) return;
  const size_t r = (size_t)z * ncol + col;
  T* o = static_cast<T*>(a.part) + ((size_t)(a.split0 + blockIdx.y) * a.N + r) * a.vstride + rhs * a.Cfull;
#pragma unroll
  for (int c = 0; c < C; ++c) o[c] = std::is_same<T, float>::value ? acc[c] : acc[c] * (T)kMonic.N[c];
}

template <int L>
cudaError_t launch_dirs(const ColArgs& a, int fp64, cudaStream_t st, int* occ) {
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, fp64 ? k_pair_dirs<L, double> : k_pair_dirs<L, float>,
                                                                PD_CTA, 0);
  const int kb = 32 * a.group, warps = (a.nx * a.ny * a.nzp + kb - 1) / kb * a.group;
  const dim3 grid((unsigned)((warps + PD_CTA / 32 - 1) / (PD_CTA / 32)), a.nsplit, a.nrhs);
  if (fp64)
    k_pair_dirs<L, double><<<grid, PD_CTA, 0, st>>>(a);
  else
    k_pair_dirs<L, float><<<grid, PD_CTA, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t rte_launch_rows_rot(const double* w, void* rows, const double* M, const int* islot, int N, int nb, int pitch,
                                int Cfull, int fp64, cudaStream_t st) {
  const long long n = (long long)N * nb * Cfull;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (fp64)
    k_rows_rot<double><<<blocks, 256, 0, st>>>(w, static_cast<double*>(rows), M, islot, N, nb, pitch, Cfull);
  else
    k_rows_rot<float><<<blocks, 256, 0, st>>>(w, static_cast<float*>(rows), M, islot, N, nb, pitch, Cfull);
  return cudaGetLastError();
}

cudaError_t rte_launch_sums_rot(const FlatArgs& a, int LA, int fp64, cudaStream_t st) {
  const int per = 256 / a.Cfull;
  const unsigned blocks = (unsigned)(((long long)a.N * a.nb + per - 1) / per);
  if (fp64)
    k_sums_rot<double><<<blocks, per * a.Cfull, 0, st>>>(a, (LA + 1) * (LA + 1));
  else
    k_sums_rot<float><<<blocks, per * a.Cfull, 0, st>>>(a, (LA + 1) * (LA + 1));
  return cudaGetLastError();
}

size_t rte_dirs_bytes(int nx, int ny, int nz, int L, int fp64) {
  return (size_t)(2 * nx - 1) * (2 * ny - 1) * (2 * nz - 1) * (fp64 || L >= 7 ? sizeof(double4) : sizeof(float4));
}

// FP32 launches of a lower order than the context's (l = 0 passes) read its table: U_0 needs no direction.
cudaError_t rte_launch_dirs_table(int nx, int ny, int nz, double dx, double dy, double dz, int transpose, int L, int fp64,
                                  void* tab, cudaStream_t st) {
  const int n = (2 * nx - 1) * (2 * ny - 1) * (2 * nz - 1), blocks = (n + 255) / 256;
  if (fp64 || L >= 7)
    k_dirs_table<double4, double><<<blocks, 256, 0, st>>>(nx, ny, nz, dx, dy, dz, transpose, static_cast<double4*>(tab));
  else
    k_dirs_table<float4, float><<<blocks, 256, 0, st>>>(nx, ny, nz, dx, dy, dz, transpose, static_cast<float4*>(tab));
  return cudaGetLastError();
}

cudaError_t rte_launch_pair_dirs(const ColArgs& a, int LA, int fp64, cudaStream_t st, int* occ) {
  switch (LA) {
    case 0: return launch_dirs<0>(a, fp64, st, occ);
    case 1: return launch_dirs<1>(a, fp64, st, occ);
    case 2: return launch_dirs<2>(a, fp64, st, occ);
    case 3: return launch_dirs<3>(a, fp64, st, occ);
    case 4: return launch_dirs<4>(a, fp64, st, occ);
    case 5: return launch_dirs<5>(a, fp64, st, occ);
    case 6: return launch_dirs<6>(a, fp64, st, occ);
    case 7: return launch_dirs<7>(a, fp64, st, occ);
  }
  return cudaErrorInvalidValue;
}

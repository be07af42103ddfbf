// rte_kernels.cu -- sm_100a kernels of the Neumann-series RTE term W <- D A W: epilogue, self-voxel term, sources,
// images, detectors, tangent and adjoint passes, the uniform-medium convolution.
//
// The attenuation operator A of the reference (FisherInfo_IO/src/kernels.cu:151-418,
// compute_diagonal_abs + compute_propabs + scale_dist_dev, and prop_scat_dev for D) is
// computed here in a REAL spherical-harmonic basis (the host converts at the boundary):
//
//   out[r,c] = sum_{r' != r, |r-r'| < propThresh} R_c(w) k(r,r') sum_c' R_c'(w) W[r',c']
//            + (dV/cm) sum_c' Dself_cc'(mu_t(r)) W[r,c'],
//   w = (r - r')/|r - r'|,  k = exp(-tau(r,r')) dV / (cm |r - r'|^2),
//
// then D multiplies coefficient (l,m) by scat[l] * mu_s(r).  The sum over pairs is in rte_column.cu, k in
// rte_store.cu; the pair sums arrive here as chunk sums that the epilogue adds in a fixed order.  The chunks are a rule
// of the grid and the order for FP64 and small grids, which makes results reproducible bit for bit; mixed launches on
// 4096 voxels and more take theirs from a timing once per process (plan_columns).
//
// Path integrals follow mu_int (FisherInfo_IO/src/kernels.cu:50-148): a Siddon walk
// between voxel centres whose axis crossings are ordered here with exact integer
// arithmetic (crossing n on an axis with |delta| = D sits at alpha = (2n+1)/(2D)).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <string.h>

#include <algorithm>

#include <type_traits>

#include "rte_device.cuh"
#include "rte_internal.h"

struct ScatTab {
  double v[RTE_MAX_L + 1];
};

__constant__ ShTables c_sh;
cudaError_t rte_upload_sh_tables(const ShTables& t) { return cudaMemcpyToSymbol(c_sh, &t, sizeof(ShTables)); }

// Real orthonormal SH R_lm at the unit direction (x, y, z), index l*l + l + m.
// R_l0 = q_l^0(z), R_l,+m = q_l^m(z) Re((x+iy)^m), R_l,-m = q_l^m(z) Im((x+iy)^m), with the
// normalised associated-Legendre polynomials q (Condon-Shortley phase included) from the
// upward recurrence in l.  No trigonometric calls.
template <int L>
__device__ __forceinline__ void sh_eval(double x, double y, double z, double* R) {
  double cmv = 1.0, smv = 0.0;
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    if (m == 1) {
      cmv = x;
      smv = y;
    } else if (m > 1) {
      double c2 = cmv * x - smv * y;
      double s2 = cmv * y + smv * x;
      cmv = c2;
      smv = s2;
    }
    double q2 = 0.0, q1 = c_sh.Q0[m];
    if (m == 0) {
      R[0] = q1;
    } else {
      R[m * m + 2 * m] = q1 * cmv;
      R[m * m] = q1 * smv;
    }
#pragma unroll
    for (int l = m + 1; l <= L; ++l) {
      const int id = l * (l + 1) / 2 + m;
      const double A = c_sh.A[id];
      double q;
      if (l == m + 1) {
        q = (A * z) * q1;
      } else {
        q = (A * z) * q1 - c_sh.B[id] * q2;
      }
      q2 = q1;
      q1 = q;
      if (m == 0) {
        R[l * l + l] = q;
      } else {
        R[l * l + l + m] = q * cmv;
        R[l * l + l - m] = q * smv;
      }
    }
  }
}

#include "rte_walk.cuh"

// ---------------------------------------------------------------------------------------------
// Plain FP64 pair operator with exact directions, every path integral walked: for callers without room for
// kernel or angle tables (rte_noalloc.cu).  One thread per destination voxel, sources streamed through shared
// memory (the warp reads the same source at the same time); `chunk` sources per blockIdx.y.
template <int LA>
__global__ void __launch_bounds__(RTE_PAIR_THREADS) k_pair_fp64(PairArgs a) {
  constexpr int C = (LA + 1) * (LA + 1), TS = RTE_PAIR_TS;
  __shared__ double sW[TS * C];
  const int tid = threadIdx.x;
  const int slot = blockIdx.x * RTE_PAIR_THREADS + tid;
  const bool act = slot < a.N;
  const int r = act ? a.perm[slot] : 0;
  const int plane = a.nx * a.ny;
  const int i = r / plane, j = (r / a.nx) % a.ny, k = r % a.nx;
  double acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0.0;
  const int sb = blockIdx.y * a.chunk;
  const int se = min(a.N, sb + a.chunk);
  for (int s0 = sb; s0 < se; s0 += TS) {
    const int ns = min(TS, se - s0);
    __syncthreads();
    for (int q = tid; q < ns * C; q += RTE_PAIR_THREADS) {
      const int sv = q / C, c = q - sv * C;
      sW[q] = a.Win[(size_t)(s0 + sv) * a.Cfull + c];
    }
    __syncthreads();
    if (!act) continue;
    int kp = s0 % a.nx, jp = (s0 / a.nx) % a.ny, ip = s0 / plane;
    for (int sv = 0; sv < ns; ++sv) {
      if (s0 + sv != r) {
        const double ddx = (double)(k - kp) * a.dx, ddy = (double)(j - jp) * a.dy, ddz = (double)(i - ip) * a.dz;
        const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
        const double dist = sqrt(d2);
        if (dist < a.prop_thresh) {
          const double inv = 1.0 / dist;
          double R[C];
          sh_eval<LA>(ddx * inv, ddy * inv, ddz * inv, R);
          double S = 0.0;
#pragma unroll
          for (int c = 0; c < C; ++c) S = fma(R[c], sW[sv * C + c], S);
          int Q;
          const double ps = path_sum<double, double>(i, j, k, ip, jp, kp, a.mut, a.nx, plane, Q);
          const double t = exp(-ps * dist / (double)Q) * a.kscale / d2 * S;
#pragma unroll
          for (int c = 0; c < C; ++c) acc[c] = fma(R[c], t, acc[c]);
        }
      }
      if (++kp == a.nx) {
        kp = 0;
        if (++jp == a.ny) {
          jp = 0;
          ++ip;
        }
      }
    }
  }
  if (act) {
    double* o = a.part + ((size_t)blockIdx.y * a.N + r) * a.Cfull;
#pragma unroll
    for (int c = 0; c < C; ++c) o[c] = acc[c];
  }
}

// q (rows qstride apart) = scat_l (mu_s T + dmu_s out): the tangent right-hand side D dA S + dD A S
__global__ void k_tangent_rhs(double* q, int qstride, const double* T, const double* out, const double* mus,
                              const double* dmus, ScatTab sc, int N, int L) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int C = (L + 1) * (L + 1);
  if (t >= (long long)N * C) return;
  const int r = (int)(t / C), c = (int)(t % C);
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  q[(size_t)r * qstride + c] = sc.v[l] * (mus[r] * T[t] + dmus[r] * out[t]);
}

__global__ void k_scatter_add(double* dst, int dstride, const int* idx, const double* vals, int n, int C) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * C) return;
  dst[(size_t)idx[t / C] * dstride + t % C] += vals[t];
}

// dst [N][C] = a (rows astride apart) + b [N][C]
__global__ void k_strided_add(double* dst, const double* a, int astride, const double* b, int N, int C) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * C) return;
  const int r = (int)(t / C), c = (int)(t % C);
  dst[t] = a[(size_t)r * astride + c] + b[t];
}

// Weight of real coefficient c in the reference stop rule's layer sum, sum over m of Re(w_lm) in the
// complex basis (dist.cu:1143-1152): for a real function R_l0 + sqrt2 R_l,m (even m > 0); for the
// imaginary part f2 of a complex function (w = w1 + i w2, Re(i w2_lm) = -Im(w2_lm)) sqrt2 R_l,-m for
// odd m > 0.
__device__ __forceinline__ double stop_weight(int c, bool imag) {
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  const int m = c - l * l - l;
  if (imag) return (m < 0 && ((-m) & 1)) ? 1.4142135623730951 : 0.0;
  return m == 0 ? 1.0 : ((m > 0 && (m % 2) == 0) ? 1.4142135623730951 : 0.0);
}

// ---------------------------------------------------------------------------------------------
// Self-voxel term (compute_diagonal_abs, FisherInfo_IO/src/kernels.cu:151-178, and its dV scale) of voxel r,
// right-hand side b, coefficient c: scale * sum_c' D(mu_t(r))[c][c'] W[r][b][c'].  D is symmetric and read by
// columns, so neighbouring c load neighbouring entries.  FIM model: voxels with mu_t == 0 (tissue 0) get nothing.
// Complex mu_t = mu_t + i kappa (the CPU package's (1 - exp(-mu_t beta)) / mu_t, Kernels_selfsub.c:927-946): even b
// is the real, odd b the imaginary row of a pair.
__device__ __forceinline__ double self_term(const SelfArgs& a, int r, int b, int c, int nb, int Cfull, int Cact) {
  const double* w = a.W + ((size_t)r * nb + b) * Cfull;
  const double mu = a.mut[r];
  if (a.kappa != 0.0) {
    const double* w0 = a.W + ((size_t)r * nb + (b & ~1)) * Cfull;
    const double* w1 = w0 + Cfull;
    double ur = 0.0, ui = 0.0;
    if (a.idx) {
      const size_t row = (size_t)a.idx[r] * Cfull * Cfull + c;
      const double* Dr = a.lut + row;
      const double* Di = a.lut_im + row;
      for (int cp = 0; cp < Cact; ++cp) {
        const double dr = __ldg(Dr + cp * Cfull), di = __ldg(Di + cp * Cfull), x0 = __ldg(w0 + cp), x1 = __ldg(w1 + cp);
        ur = fma(dr, x0, fma(-di, x1, ur));
        ui = fma(dr, x1, fma(di, x0, ui));
      }
    } else {  // Horner in the complex mu: u <- mu u + M_k w
      for (int kk = a.K - 1; kk >= 0; --kk) {
        const double* M = a.mom + (size_t)kk * Cfull * Cfull + c;
        double t0 = 0.0, t1 = 0.0;
        for (int cp = 0; cp < Cact; ++cp) {
          const double m = __ldg(M + cp * Cfull);
          t0 = fma(m, __ldg(w0 + cp), t0);
          t1 = fma(m, __ldg(w1 + cp), t1);
        }
        const double nr = mu * ur - a.kappa * ui + t0, ni = mu * ui + a.kappa * ur + t1;
        ur = nr;
        ui = ni;
      }
    }
    return a.scale * ((b & 1) ? ui : ur);
  }
  if (a.air_no_self && mu == 0.0) return 0.0;
  double u = 0.0;
  if (a.idx) {
    const double* D = a.lut + (size_t)a.idx[r] * Cfull * Cfull + c;
    for (int cp = 0; cp < Cact; ++cp) u = fma(__ldg(D + cp * Cfull), __ldg(w + cp), u);
  } else {  // D(mu) = sum_k mu^k M_k; its derivative sum_k k mu^(k-1) M_k, both by Horner
    const bool der = a.dmut != nullptr;
    for (int kk = a.K - 1; kk >= (der ? 1 : 0); --kk) {
      const double* M = a.mom + (size_t)kk * Cfull * Cfull + c;
      double tk = 0.0;
      for (int cp = 0; cp < Cact; ++cp) tk = fma(__ldg(M + cp * Cfull), __ldg(w + cp), tk);
      u = fma(mu, u, der ? (double)kk * tk : tk);
    }
  }
  if (a.dmut) u *= a.dmut[r];
  return a.scale * u;
}

// Epilogue: self-voxel term, chunk sums, scatter; write the next term (and its rows for the next pair launch),
// accumulate the running sum and the norms used by the stop rules.  One thread per (voxel, right-hand side,
// coefficient) element, grid-stride, so every stream (chunk sums, outputs, running sum) is read and written
// coalesced; the four norms are reduced per block and added atomically.  Bound by loads of the self-term table
// (2 C per element, from L1 and L2) and of the chunk sums.  Measured per term, self term and epilogue together (by the
// number of chunks): 171 -> 90 us at 33^3 L=5, 448 -> 290 us with four right-hand sides, 310 -> 79 us at 25^3 L=7 against a self-term launch of
// its own that read rows of D.  Coefficients above (LA+1)^2 are written as 0.
__global__ void __launch_bounds__(256) k_epilogue(EpiArgs a, int Cact) {
  const int nb = a.nb > 0 ? a.nb : 1;
  const int vstride = nb * a.Cfull;
  const size_t total = (size_t)a.N * vstride, NV = (size_t)a.N * vstride;
  const int plane = a.nx * a.ny;
  double w2 = 0.0, s2 = 0.0, lw = 0.0, ls = 0.0;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int r = total < (1ull << 32) ? (int)((unsigned)t / (unsigned)vstride) : (int)(t / vstride);
    const int e = (int)(t - (size_t)r * vstride), b = nb == 1 ? 0 : e / a.Cfull, c = e - b * a.Cfull;
    int l = 0;
    while ((l + 1) * (l + 1) <= c) ++l;
    double x = 0.0;
    if (c < Cact) {
      x = a.self.W ? self_term(a.self, r, b, c, nb, a.Cfull, Cact) : 0.0;
      if (a.partf) {  // FP32 chunk sums: FP64 sum over the chunks, then N_c
        double u = 0.0;
        for (int q = 0; q < a.S; ++q) u += (double)a.partf[(size_t)q * NV + t];
        x = fma(u, kMonic.N[c], x);
      } else {
        for (int q = 0; q < a.S; ++q) x += a.part[(size_t)q * NV + t];
      }
      if (a.flag_scat) x *= a.scat[l] * a.mus[r];
    }
    a.Wout[t] = x;
    // the column kernels read N_c W_c (rte_trig.cuh)
    if (a.rows) {
      const size_t o = ((size_t)b * a.N + a.islot[r]) * a.pitch + c;
      if (a.rows64)
        static_cast<double*>(a.rows)[o] = x * kMonic.N[c];
      else
        static_cast<float*>(a.rows)[o] = (float)(x * kMonic.N[c]);
    }
    w2 += x * x;
    double sv = 0.0;
    if (a.sum) {
      sv = a.sum[t] + x;
      a.sum[t] = sv;
      s2 += sv * sv;
    }
    if (r / plane == a.nz - 1) {  // the reference stop rule's layer
      const double wgt = stop_weight(c, a.cplx && (b & 1));
      lw += wgt * x;
      ls += wgt * sv;
    }
  }
  // block reduction of the four norms
  __shared__ double red[4][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double vals[4] = {w2, s2, lw, ls};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double x = vals[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[q][wid] = x;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double x = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += red[threadIdx.x][w];
    atomicAdd(a.red + threadIdx.x, x);
  }
}

// Exitance images of the z = nZ-1 and z = 0 faces from the m = 0 coefficients
// (FisherInfo_IO/src/dist.cu:103-161, 229-268; the per-l weights come from the host).
__global__ void k_images(ImgArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.nx * a.ny) return;
  const double* out_im = a.out_im;
  const size_t rt = (size_t)(a.nz - 1) * a.nx * a.ny + p, rr = (size_t)p;
  double t = 0.0, f = 0.0, ti = 0.0, fi = 0.0;
  for (int l = 0; l <= a.L; ++l) {
    const int c = l * l + l;
    t += a.wt[l] * a.out[rt * a.vstride + c];
    f += a.wr[l] * a.out[rr * a.vstride + c];
    if (out_im) {
      ti += a.wt[l] * out_im[rt * a.vstride + c];
      fi += a.wr[l] * out_im[rr * a.vstride + c];
    }
  }
  if (a.fball) {
    t += a.fball[(size_t)a.nx * a.ny + p];
    f += a.fball[p];
  }
  if (a.fball_im) {
    ti += a.fball_im[(size_t)a.nx * a.ny + p];
    fi += a.fball_im[p];
  }
  if (a.trans) {
    a.trans[2 * p] = t;
    a.trans[2 * p + 1] = ti;
  }
  if (a.ref) {
    a.ref[2 * p] = f;
    a.ref[2 * p + 1] = fi;
  }
}

// Collimated-beam source xi = D A xi_beam on the pencil columns (one thread per column), with the
// ballistic transmission of each column.  FisherInfo_IO/src/dist.cu:66-101 (product of per-layer
// attenuations) and, for kind 2, CPU package/src/Dist.c:1077-1128 (attenuation from the absolute
// depth of the voxel, normalised by the number of columns).
__global__ void k_source(SrcArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.ncols) return;
  const int p = a.cols[q];
  const int plane = a.nx * a.ny;
  const int axis = a.face / 2;  // 0: along z, 1: along y, 2: along x
  const bool up = (a.face & 1) == 0;
  int n, base, stride, row, col;
  if (axis == 0) {
    n = a.nz;
    base = p;
    stride = plane;
  } else if (axis == 1) {
    n = a.ny;
    row = p / a.nx;  // i
    col = p % a.nx;  // k
    base = row * plane + col;
    stride = a.nx;
  } else {
    n = a.nx;
    row = p / a.ny;  // i
    col = p % a.ny;  // j
    base = row * plane + col * a.nx;
    stride = 1;
  }
  // attenuation with mu_t + i kappa (kappa = 0: the steady state); complex values as (re, im)
  const double kap = a.kappa;
  auto cexpm = [kap](double m, double x, double& re, double& im) {  // exp(-(m + i kap) x)
    const double e = exp(-m * x);
    double sn = 0.0, cs = 1.0;
    if (kap != 0.0) sincos(kap * x, &sn, &cs);
    re = e * cs;
    im = -e * sn;
  };
  double attr = 1.0, atti = 0.0, mt = 0.0;
  for (int t = 0; t < n; ++t) {
    const size_t r = (size_t)base + (size_t)(up ? t : n - 1 - t) * stride;
    mt = a.mut[r];
    const double ms = a.mus[r];
    double vr, vi, er, ei;
    cexpm(mt, a.dlen, er, ei);
    if (a.kind == 2) {  // absolute depth of the voxel top (z- entry only)
      const double tz = (double)t * a.dz + a.z_min + a.dz / 2.0 - a.dz / 2.0;
      double e1r, e1i, e2r, e2i;
      cexpm(mt, tz, e1r, e1i);
      cexpm(mt, tz + a.dz, e2r, e2i);
      vr = e1r - e2r;
      vi = e1i - e2i;
    } else {  // att * (1 - exp(-mu dlen))
      vr = attr * (1.0 - er) + atti * ei;
      vi = atti * (1.0 - er) - attr * ei;
    }
    const double nr = attr * er - atti * ei, ni = attr * ei + atti * er;
    attr = nr;
    atti = ni;
    // amp = ms / (mt + i kap) * v / dV
    double ar, ai = 0.0;
    if (kap == 0.0) {
      ar = ms / mt * vr / a.dV;
    } else {
      const double den = mt * mt + kap * kap;
      ar = ms * (mt * vr + kap * vi) / den / a.dV;
      ai = ms * (mt * vi - kap * vr) / den / a.dV;
    }
    for (int c = 0; c < a.Cfull; ++c)
      if (a.coef[c] != 0.0) {
        a.W[r * a.vstride + c] += ar * a.coef[c];
        if (kap != 0.0) a.W[r * a.vstride + a.Cfull + c] += ai * a.coef[c];
      }
  }
  // exit face = the opposite face, same in-face pixel
  const int ef = a.face ^ 1;
  const size_t a0 = (size_t)a.nx * a.ny, a1 = (size_t)a.nz * a.nx, a2 = (size_t)a.nz * a.ny;
  const size_t off[6] = {0, a0, 2 * a0, 2 * a0 + a1, 2 * a0 + 2 * a1, 2 * a0 + 2 * a1 + a2};
  double br, bi;
  if (a.kind == 2) {
    const double zs = (double)(a.nz - 1) * a.dz + a.z_min + a.dz / 2.0;
    cexpm(mt, zs + a.dz / 2.0, br, bi);
    br *= a.scale;
    bi *= a.scale;
  } else {
    br = a.mag * attr;
    bi = a.mag * atti;
  }
  a.fball[off[ef] + p] = br;
  if (a.fball_im) a.fball_im[off[ef] + p] = bi;
}

// mu_t = mu_a + mu_s (FP64 in voxel and column order, FP32 in column order), mu_s copy, and max(mu_t) into red_max (>= 0 values,
// so the bit pattern orders like the value).
__global__ void k_medium(const double* mua, const double* mus, double* mut, double* mus_out, double* mutc,
                         float* mutfc, const int* islot, int N, double* red_max) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (r < N) {
    m = mua[r] + mus[r];
    mut[r] = m;
    mutc[islot[r]] = m;
    mutfc[islot[r]] = (float)m;
    if (mus_out != mus) mus_out[r] = mus[r];
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax((unsigned long long*)red_max, (unsigned long long)__double_as_longlong(m));
}

// FMA throughput probe (roofline denominator for the CUDA-core-bound kernels): 8 independent FMA
// chains per thread; the result is written so the work cannot be removed.  k_fma2_peak does the
// same with packed f32x2 FMAs (two FP32 FMAs per instruction).
__global__ void k_fma2_peak(int iters, float* sink) {
  f2_t a[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) a[q] = f2_pack((float)(threadIdx.x + q) * 1e-3f, (float)(threadIdx.x + 2 * q) * 1e-3f);
  const f2_t b = f2_pack(0.999999f, 0.999998f), c = f2_pack(1e-7f, 2e-7f);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = f2_fma(a[q], b, c);
  }
  float s = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    float lo, hi;
    f2_unpack(a[q], lo, hi);
    s += lo + hi;
  }
  if (s == -1.2345f) sink[blockIdx.x] = s;
}

// k_fma2_fresh_peak: packed FMAs whose three operands are all distinct registers (none shared with the
// neighbouring instructions), the operand pattern of the pair kernels' source-row dot products.
__global__ void k_fma2_fresh_peak(int iters, float* sink) {
  f2_t a[12], x[12], y[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    a[q] = f2_pack((float)(threadIdx.x + q) * 1e-3f, (float)(threadIdx.x + 2 * q) * 1e-3f);
    x[q] = f2_pack(0.9999f + (float)q * 1e-7f, 0.9998f + (float)q * 1e-7f);
    y[q] = f2_pack(1e-7f * (float)(q + 1) + (float)threadIdx.x * 1e-9f, 2e-7f * (float)(q + 1));
  }
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int q = 0; q < 12; ++q) a[q] = f2_fma(x[q], a[q], y[q]);
  }
  float s = 0.f;
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    float lo, hi;
    f2_unpack(a[q], lo, hi);
    s += lo + hi;
  }
  if (s == -1.2345f) sink[blockIdx.x] = s;
}

template <typename T>
__global__ void k_fma_peak(int iters, float* sink) {
  T a[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) a[q] = (T)(threadIdx.x + q) * (T)1e-3;
  const T b = (T)0.999999, c = (T)1e-7;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = fma(a[q], b, c);
  }
  T s = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += a[q];
  if (s == (T)-1.2345) sink[blockIdx.x] = (float)s;
}

// ---------------------------------------------------------------------------------------------
// Detectors and the adjoint gradient.
// Face pixels: z-(ny*nx) z+(ny*nx) y-(nz*nx) y+(nz*nx) x-(nz*ny) x+(nz*ny), row-major.
__device__ __forceinline__ void face_pixel(int q, int nx, int ny, int nz, int& f, int& p, int& r) {
  const int a0 = nx * ny, a1 = nz * nx, a2 = nz * ny;
  const int off[6] = {0, a0, 2 * a0, 2 * a0 + a1, 2 * a0 + 2 * a1, 2 * a0 + 2 * a1 + a2};
  f = 5;
  for (int t = 1; t < 6; ++t)
    if (q < off[t]) {
      f = t - 1;
      break;
    }
  p = q - off[f];
  if (f < 2) {  // p = j*nx + k
    const int i = f == 0 ? 0 : nz - 1;
    r = i * nx * ny + p;
  } else if (f < 4) {  // p = i*nx + k
    const int i = p / nx, k = p % nx, j = f == 2 ? 0 : ny - 1;
    r = (i * ny + j) * nx + k;
  } else {  // p = i*ny + j
    const int i = p / ny, j = p % ny, k = f == 4 ? 0 : nx - 1;
    r = (i * ny + j) * nx + k;
  }
}

__global__ void k_face_flux(FaceArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int total = 2 * (a.nx * a.ny + a.nz * a.nx + a.nz * a.ny);
  if (q >= total) return;
  int f, p, r;
  face_pixel(q, a.nx, a.ny, a.nz, f, p, r);
  const double* h = a.h + f * a.Cfull;
  const double* o = a.out + (size_t)r * a.vstride;
  double J = 0.0;
  for (int c = 0; c < a.Cfull; ++c) J = fma(h[c], o[c], J);
  if (a.fball) J += a.fball[q];
  a.J[q] = J;
}

// e[r][c] += rho(pixel) h_f[c] for every face pixel (edge voxels belong to several faces)
__global__ void k_adjoint_seed(FaceArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int total = 2 * (a.nx * a.ny + a.nz * a.nx + a.nz * a.ny);
  if (q >= total) return;
  const double rho = a.rho[q];
  if (rho == 0.0) return;
  int f, p, r;
  face_pixel(q, a.nx, a.ny, a.nz, f, p, r);
  for (int c = 0; c < a.Cfull; ++c) atomicAdd(a.e + (size_t)r * a.Cfull + c, rho * a.h[f * a.Cfull + c]);
}

// x *= (-1)^l: the parity of the real SH, R(-w) = (-1)^l R(w); the transpose of the pair operator
// is P A P.
__global__ void k_parity(double* x, int N, int L, int vstride) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int C = (L + 1) * (L + 1);
  if (t >= (long long)N * C) return;
  const int r = (int)(t / C), c = (int)(t % C);
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  if (l & 1) x[(size_t)r * vstride + c] = -x[(size_t)r * vstride + c];
}

// out[r][c] = mask[r] ? fac[l(c)] * in[r][c] : 0 -- the region-restricted tangent sources of the
// reference's inverse and Fisher mains (compute_grad_rte.cu:288-363, rte_fim.cu:253-273).
__global__ void k_masked_scale(const double* in, double* out, const uint8_t* mask, ScatTab fac, int N, int L) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int C = (L + 1) * (L + 1);
  if (t >= (long long)N * C) return;
  const int r = (int)(t / C), c = (int)(t % C);
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  out[t] = mask[r] ? fac.v[l] * in[t] : 0.0;
}

// Per voxel: ga[r] = sum_c fa[l(c)] lam[r][c] out[r][c], gs likewise with fs -- the reference's tangent
// sources (-C out for mu_a, (-C + g^l) out for mu_s, compute_grad_rte.cu:296-299, 343-350) paired with
// an adjoint field.
__global__ void k_tangent_pair_dots(const double* lam, const double* out, ScatTab fa, ScatTab fs, int N, int L,
                                    double* ga, double* gs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int C = (L + 1) * (L + 1);
  const size_t b = (size_t)r * C;
  double a = 0.0, s = 0.0;
  for (int l = 0; l <= L; ++l)
    for (int c = l * l; c < (l + 1) * (l + 1); ++c) {
      const double p = lam[b + c] * out[b + c];
      a = fma(fa.v[l], p, a);
      s = fma(fs.v[l], p, s);
    }
  ga[r] = a;
  gs[r] = s;
}

__global__ void k_axpy(double* y, const double* x, double alpha, size_t n) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) y[t] = fma(alpha, x[t], y[t]);
}

// y = e + D lambda, D = scat_l mu_s(r)
__global__ void k_y_field(double* y, const double* e, const double* lam, const double* mus, ScatTab sc, int N, int L,
                          int Cfull) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * Cfull) return;
  const int r = (int)(t / Cfull), c = (int)(t % Cfull);
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  y[t] = e[t] + (l <= L ? sc.v[l] : 0.0) * mus[r] * lam[t];
}

__host__ __device__ constexpr int l_of_c(int c) {
  int l = 0;
  while ((l + 1) * (l + 1) <= c) ++l;
  return l;
}

// Per-voxel parts of the gradient: the scatter D (d/dmu_s: lambda . scat_l . (A S)) and the
// self-voxel term (d/dmu_t: (dV/cm) y . dDself/dmu S).
__global__ void k_grad_local(GradLocalArgs a) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.N) return;
  const size_t b = (size_t)r * a.Cfull;
  double gs = 0.0;
  for (int c = 0; c < a.Cact; ++c) {
    int l = 0;
    while ((l + 1) * (l + 1) <= c) ++l;
    gs = fma(a.lam[b + c] * a.scat[l], a.out[b + c], gs);
  }
  a.gs[r] += gs;
  const double mu = a.mut[r];
  if (a.air_no_self && mu == 0.0) return;
  double gt = 0.0;
  for (int c = 0; c < a.Cact; ++c) {
    double u = 0.0;
    if (a.idx) {
      const double* D = a.dlut + ((size_t)a.idx[r] * a.Cfull + c) * a.Cfull;
      for (int cp = 0; cp < a.Cact; ++cp) u = fma(D[cp], a.S[b + cp], u);
    } else {
      // d/dmu sum_k mu^k M_k = sum_{k>=1} k mu^(k-1) M_k
      for (int kk = a.K - 1; kk >= 1; --kk) {
        const double* M = a.mom + ((size_t)kk * a.Cfull + c) * a.Cfull;
        double t = 0.0;
        for (int cp = 0; cp < a.Cact; ++cp) t = fma(M[cp], a.S[b + cp], t);
        u = fma(mu, u, (double)kk * t);
      }
    }
    gt = fma(a.y[b + c], u, gt);
  }
  a.gt[r] += a.scale * gt;
}

// Complex reference basis <-> real basis.  w = w1 + i w2 with w1, w2 the coefficient sets of
// real functions (w_{l,-m} = (-1)^m conj(w_{l,m})).  u_l0 = Re(w_l0), u_l,m = sqrt2 Re(w_lm),
// u_l,-m = -sqrt2 Im(w_lm) (m > 0).  red[0] accumulates ||u2||^2.
__global__ void k_to_real(const double* __restrict__ w, double* u1, double* u2, int N, int L, double* red,
                          int ostride) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double n2 = 0.0;
  if (r < N) {
    const int C = (L + 1) * (L + 1);
    // u1/u2 rows are ostride apart (a complex right-hand side's real and imaginary rows interleaved)
    u1 += (size_t)r * ostride - (size_t)r * C;
    if (u2) u2 += (size_t)r * ostride - (size_t)r * C;
    const double s2 = 1.4142135623730951;
    for (int l = 0; l <= L; ++l) {
      const int c0 = l * l + l;
      const double re0 = w[2 * ((size_t)r * C + c0)], im0 = w[2 * ((size_t)r * C + c0) + 1];
      u1[(size_t)r * C + c0] = re0;
      if (u2) u2[(size_t)r * C + c0] = im0;
      n2 += im0 * im0;
      for (int m = 1; m <= l; ++m) {
        const double sg = (m & 1) ? -1.0 : 1.0;
        const size_t ip = (size_t)r * C + c0 + m, in = (size_t)r * C + c0 - m;
        const double rp = w[2 * ip], mp = w[2 * ip + 1], rn = w[2 * in], mn = w[2 * in + 1];
        // w1 = (w + P w)/2, P w_lm = (-1)^m conj(w_l,-m)
        const double r1 = 0.5 * (rp + sg * rn), i1 = 0.5 * (mp - sg * mn);
        // w2 = (w - P w)/(2i)
        const double dr = rp - sg * rn, di = mp + sg * mn;
        const double r2 = 0.5 * di, i2 = -0.5 * dr;
        u1[ip] = s2 * r1;
        u1[in] = -s2 * i1;
        if (u2) {
          u2[ip] = s2 * r2;
          u2[in] = -s2 * i2;
        }
        n2 += r2 * r2 + i2 * i2;
      }
    }
  }
  if (red) {
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    if ((threadIdx.x & 31) == 0 && n2 != 0.0) atomicAdd(red, n2);
  }
}

__global__ void k_to_cplx(const double* __restrict__ u1, const double* __restrict__ u2, double* w, int N, int L,
                          int ustride) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int C = (L + 1) * (L + 1);
  // u1/u2 rows are ustride apart (several right-hand sides interleaved); w rows are C apart
  u1 += (size_t)r * ustride - (size_t)r * C;
  if (u2) u2 += (size_t)r * ustride - (size_t)r * C;
  const double is2 = 0.70710678118654752;
  for (int l = 0; l <= L; ++l) {
    const int c0 = l * l + l;
    const size_t i0 = (size_t)r * C + c0;
    // w = w1 + i w2
    w[2 * i0] = u1[i0];
    w[2 * i0 + 1] = u2 ? u2[i0] : 0.0;
    for (int m = 1; m <= l; ++m) {
      const double sg = (m & 1) ? -1.0 : 1.0;
      const size_t ip = i0 + m, in = i0 - m;
      // w1_lm = (a - i b)/sqrt2, w1_l,-m = (-1)^m (a + i b)/sqrt2 with a = u_l,m, b = u_l,-m
      const double a1 = u1[ip], b1 = u1[in];
      double wr_p = a1 * is2, wi_p = -b1 * is2, wr_n = sg * a1 * is2, wi_n = sg * b1 * is2;
      if (u2) {
        const double a2 = u2[ip], b2 = u2[in];
        // + i * w2: i(a2 - i b2)/sqrt2 = (b2 + i a2)/sqrt2 ; i * (-1)^m (a2 + i b2)/sqrt2 = (-1)^m(-b2 + i a2)/sqrt2
        wr_p += b2 * is2;
        wi_p += a2 * is2;
        wr_n += -sg * b2 * is2;
        wi_n += sg * a2 * is2;
      }
      w[2 * ip] = wr_p;
      w[2 * ip + 1] = wi_p;
      w[2 * in] = wr_n;
      w[2 * in + 1] = wi_n;
    }
  }
}

// Stop-rule sums of the layer z = nZ-1 (FisherInfo_IO/src/dist.cu:1143-1152) in the real basis;
// cplx: (real, imaginary) row pairs per voxel.
__global__ void k_layer_sums(const double* W, const double* S, int N, int nx, int ny, int nz, int Cfull,
                             double* red, int cplx) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  double lw = 0.0, ls = 0.0;
  const int np = cplx ? 2 : 1;
  if (p < nx * ny) {
    const size_t r = (size_t)(nz - 1) * nx * ny + p;
    for (int q = 0; q < np; ++q)
      for (int c = 0; c < Cfull; ++c) {
        const double wgt = stop_weight(c, q == 1);
        const size_t e = (r * np + q) * Cfull + c;
        lw += wgt * W[e];
        ls += wgt * S[e];
      }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lw += __shfl_xor_sync(0xffffffffu, lw, o);
    ls += __shfl_xor_sync(0xffffffffu, ls, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(red + 2, lw);
    atomicAdd(red + 3, ls);
  }
}

// ---------------------------------------------------------------------------------------------
// launchers

cudaError_t rte_launch_pair_fp64(const PairArgs& a, int LA, cudaStream_t st) {
  dim3 grid((a.N + RTE_PAIR_THREADS - 1) / RTE_PAIR_THREADS, a.nsplit);
  switch (LA) {
    case 0: k_pair_fp64<0><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 1: k_pair_fp64<1><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 2: k_pair_fp64<2><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 3: k_pair_fp64<3><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 4: k_pair_fp64<4><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 5: k_pair_fp64<5><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 6: k_pair_fp64<6><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    case 7: k_pair_fp64<7><<<grid, RTE_PAIR_THREADS, 0, st>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t rte_launch_epilogue(const EpiArgs& a, int LA, cudaStream_t st) {
  if (LA < 0 || LA > RTE_MAX_L) return cudaErrorInvalidValue;
  const size_t total = (size_t)a.N * (a.nb > 0 ? a.nb : 1) * a.Cfull;
  const unsigned blocks = (unsigned)std::min<size_t>((total + 255) / 256, 148 * 16);
  k_epilogue<<<blocks, 256, 0, st>>>(a, (LA + 1) * (LA + 1));
  return cudaGetLastError();
}

cudaError_t rte_launch_images(const ImgArgs& a, cudaStream_t st) {
  const int n = a.nx * a.ny;
  k_images<<<(n + 127) / 128, 128, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t rte_launch_to_real(const double* cplx, double* u1, double* u2, int N, int L, double* red,
                               cudaStream_t st, int ostride) {
  const int C = (L + 1) * (L + 1);
  k_to_real<<<(N + 127) / 128, 128, 0, st>>>(cplx, u1, u2, N, L, red, ostride > 0 ? ostride : C);
  return cudaGetLastError();
}

cudaError_t rte_launch_to_cplx(const double* u1, const double* u2, double* cplx, int N, int L, cudaStream_t st,
                               int ustride) {
  const int C = (L + 1) * (L + 1);
  k_to_cplx<<<(N + 127) / 128, 128, 0, st>>>(u1, u2, cplx, N, L, ustride > 0 ? ustride : C);
  return cudaGetLastError();
}

cudaError_t rte_launch_layer_sums(const double* W, const double* S, int N, int nx, int ny, int nz, int Cfull,
                                  double* red, cudaStream_t st, int cplx) {
  const int n = nx * ny;
  k_layer_sums<<<(n + 127) / 128, 128, 0, st>>>(W, S, N, nx, ny, nz, Cfull, red, cplx);
  return cudaGetLastError();
}

cudaError_t rte_launch_source(const SrcArgs& a, cudaStream_t st) {
  k_source<<<(a.ncols + 31) / 32, 32, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t rte_launch_medium(const double* mua, const double* mus, double* mut, double* mus_out, double* mutc, float* mutfc, const int* islot, int N, double* red_max, cudaStream_t st) {
  k_medium<<<(N + 127) / 128, 128, 0, st>>>(mua, mus, mut, mus_out, mutc, mutfc, islot, N, red_max);
  return cudaGetLastError();
}

cudaError_t rte_launch_fma_peak(int fp64, int iters, float* sink, cudaStream_t st, int blocks) {
  if (fp64 == 3)
    k_fma2_fresh_peak<<<blocks, 256, 0, st>>>(iters, sink);
  else if (fp64 == 2)
    k_fma2_peak<<<blocks, 256, 0, st>>>(iters, sink);
  else if (fp64)
    k_fma_peak<double><<<blocks, 256, 0, st>>>(iters, sink);
  else
    k_fma_peak<float><<<blocks, 256, 0, st>>>(iters, sink);
  return cudaGetLastError();
}

cudaError_t rte_launch_face_flux(const FaceArgs& a, cudaStream_t st) {
  const int total = 2 * (a.nx * a.ny + a.nz * a.nx + a.nz * a.ny);
  k_face_flux<<<(total + 127) / 128, 128, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t rte_launch_adjoint_seed(const FaceArgs& a, cudaStream_t st) {
  const int total = 2 * (a.nx * a.ny + a.nz * a.nx + a.nz * a.ny);
  k_adjoint_seed<<<(total + 127) / 128, 128, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t rte_launch_tangent_rhs(double* q, int qstride, const double* T, const double* out, const double* mus,
                                   const double* dmus, const double* scat, int N, int L, cudaStream_t st) {
  ScatTab sc;
  for (int l = 0; l <= RTE_MAX_L; ++l) sc.v[l] = l <= L ? scat[l] : 0.0;
  const long long n = (long long)N * (L + 1) * (L + 1);
  k_tangent_rhs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(q, qstride, T, out, mus, dmus, sc, N, L);
  return cudaGetLastError();
}

cudaError_t rte_launch_scatter_add(double* dst, int dstride, const int* idx, const double* vals, int n, int C,
                                   cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_scatter_add<<<(n * C + 255) / 256, 256, 0, st>>>(dst, dstride, idx, vals, n, C);
  return cudaGetLastError();
}

cudaError_t rte_launch_strided_add(double* dst, const double* a, int astride, const double* b, int N, int C,
                                   cudaStream_t st) {
  const long long n = (long long)N * C;
  k_strided_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dst, a, astride, b, N, C);
  return cudaGetLastError();
}

cudaError_t rte_launch_masked_scale(const double* in, double* out, const uint8_t* mask, const double* fac, int N,
                                    int L, cudaStream_t st) {
  ScatTab f;
  for (int l = 0; l <= RTE_MAX_L; ++l) f.v[l] = l <= L ? fac[l] : 0.0;
  const long long n = (long long)N * (L + 1) * (L + 1);
  k_masked_scale<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, mask, f, N, L);
  return cudaGetLastError();
}

cudaError_t rte_launch_parity(double* x, int N, int L, int vstride, cudaStream_t st) {
  const long long n = (long long)N * (L + 1) * (L + 1);
  k_parity<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, N, L, vstride);
  return cudaGetLastError();
}

cudaError_t rte_launch_tangent_pair_dots(const double* lam, const double* out, const double* fa, const double* fs, int N,
                                         int L, double* ga, double* gs, cudaStream_t st) {
  ScatTab a, b;
  for (int l = 0; l <= RTE_MAX_L; ++l) {
    a.v[l] = l <= L ? fa[l] : 0.0;
    b.v[l] = l <= L ? fs[l] : 0.0;
  }
  k_tangent_pair_dots<<<(N + 127) / 128, 128, 0, st>>>(lam, out, a, b, N, L, ga, gs);
  return cudaGetLastError();
}

cudaError_t rte_launch_axpy(double* y, const double* x, double alpha, size_t n, cudaStream_t st) {
  k_axpy<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y, x, alpha, n);
  return cudaGetLastError();
}

cudaError_t rte_launch_y_field(double* y, const double* e, const double* lam, const double* mus, const double* scat,
                               int N, int L, int Cfull, cudaStream_t st) {
  ScatTab sc;
  for (int l = 0; l <= RTE_MAX_L; ++l) sc.v[l] = scat[l];
  const long long n = (long long)N * Cfull;
  k_y_field<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y, e, lam, mus, sc, N, L, Cfull);
  return cudaGetLastError();
}

cudaError_t rte_launch_grad_local(const GradLocalArgs& a, cudaStream_t st) {
  k_grad_local<<<(a.N + 127) / 128, 128, 0, st>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Uniform medium: the off-diagonal operator as a convolution over displacements (host side and the
// transforms in rte_fft.cpp).  k_fft_table samples T_cc'(d) = k(d) R_c(d) R_c'(d) on the padded
// grid, k_fft_pad / k_fft_crop move fields in and out of it, k_fft_product forms the spectral
// products.
// T_cc'(d) for c <= c' (pair p in row-major upper-triangle order) on the padded grid; the padded
// index g maps to the displacement g (g < n), g - M (g > n) or none (g == n).
template <int LA, bool TABLE>
__global__ void k_fft_table(FftTabArgs a, double* T, size_t M) {
  constexpr int C = (LA + 1) * (LA + 1);
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= M) return;
  const int gx = (int)(t % a.Mx), gy = (int)((t / a.Mx) % a.My), gz = (int)(t / ((size_t)a.Mx * a.My));
  auto disp = [](int g, int n, int Mg, bool& ok) {
    if (g < n) return g;
    if (g > Mg - n) return g - Mg;
    ok = false;
    return 0;
  };
  bool ok = true;
  const int ix = disp(gx, a.nx, a.Mx, ok), iy = disp(gy, a.ny, a.My, ok), iz = disp(gz, a.nz, a.Mz, ok);
  const double ddx = ix * a.dx, ddy = iy * a.dy, ddz = iz * a.dz;
  const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
  const double dist = sqrt(d2);
  ok = ok && d2 > 0.0 && dist < a.prop_thresh;
  double R[C];
  double k = 0.0;
  if (ok) {
    k = exp(-a.mut * dist) * a.kscale / d2;
    double ux, uy, uz;
    if (TABLE) {
      table_direction(ddx, ddy, ddz, dist, ux, uy, uz);
    } else {
      ux = ddx / dist;
      uy = ddy / dist;
      uz = ddz / dist;
    }
    sh_eval<LA>(ux, uy, uz, R);
  }
  int p = 0;
#pragma unroll 1
  for (int c = 0; c < C; ++c)
#pragma unroll 1
    for (int cp = c; cp < C; ++cp, ++p)
      if (p >= a.p0 && p < a.p1) T[(size_t)(p - a.p0) * M + t] = ok ? k * R[c] * R[cp] : 0.0;
}

// W [N][vstride] (coefficient c of right-hand side b at b*Cfull + c) -> padded fields F[b*Cact + c][M]
__global__ void k_fft_pad(const double* W, int vstride, int Cfull, int Cact, int nb, FftTabArgs a, double* F,
                          size_t M) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long N = (long long)a.nx * a.ny * a.nz;
  if (t >= N * nb * Cact) return;
  const int c = (int)(t % Cact);
  const int b = (int)((t / Cact) % nb);
  const long long r = t / ((long long)Cact * nb);
  const int x = (int)(r % a.nx), y = (int)((r / a.nx) % a.ny), z = (int)(r / ((long long)a.nx * a.ny));
  F[(size_t)(b * Cact + c) * M + ((size_t)z * a.My + y) * a.Mx + x] = W[(size_t)r * vstride + (size_t)b * Cfull + c];
}

// Spectral products O_c(k) = sum_c' That_cc'(k) W_c'(k).  T_cc'(-d) = (-1)^(l+l') T_cc'(d), so each
// table spectrum is real (l + l' even) or imaginary (odd): the table holds one real number tau per
// pair and frequency (That = tau or i tau), c <= c' in row-major upper-triangle order of the full
// order.  The complex products then split into two real systems over the coefficients,
//   set 0: inputs (Re W_even, Im W_odd) -> outputs (Re O_even, Im O_odd),
//   set 1: inputs (Im W_even, Re W_odd) -> outputs (Im O_even, Re O_odd),
// with sign -1 on the even<-odd terms of set 0 and the odd<-even terms of set 1 (i * i = -1).
__device__ __forceinline__ double fft_sign(int set, bool c_even, bool cp_even) {
  if (c_even == cp_even) return 1.0;
  return (set == 0) == c_even ? -1.0 : 1.0;
}

// The two real systems of a frequency run on adjacent lanes (set = lane parity), so the pair's table
// loads are one memory transaction and the table spectrum (larger than L2 at benchmark sizes) streams
// from HBM once per right-hand side instead of once per set.  Three CTAs per SM (168 registers, a small
// spill) keep more table loads in flight than two at 255 registers: 33^3 L=5 uniform solve 23.6 -> 22.5
// ms (four CTAs: 22.4 ms with a 3 KB spill).
template <int LA>
__global__ void __launch_bounds__(128, 3) k_fft_product_reg(const double* tau, const double2* Wh, double2* Oh, int C,
                                                         int nb, size_t Mk) {
  constexpr int CA = (LA + 1) * (LA + 1);
  __shared__ double sv[CA][128];  // this thread's inputs of its set (column tid)
  const int tid = threadIdx.x;
  const size_t g = (size_t)blockIdx.x * blockDim.x + tid;
  const size_t k = g >> 1;
  const int set = (int)(g & 1);
  const bool act = k < Mk;
  double* Ohd = reinterpret_cast<double*>(Oh);
  for (int b = 0; b < nb; ++b) {
    {
      double q[CA];
#pragma unroll
      for (int c = 0; c < CA; ++c) {
        const bool ev = !(l_of_c(c) & 1);
        const double2 w = act ? Wh[(size_t)(b * CA + c) * Mk + k] : make_double2(0.0, 0.0);
        sv[c][tid] = ((set == 0) == ev) ? w.x : w.y;
        q[c] = 0.0;
      }
      if (act) {
#pragma unroll
        for (int c = 0; c < CA; ++c) {
          const size_t row = (size_t)c * C - (size_t)c * (c - 1) / 2;
          const double vc = sv[c][tid];
#pragma unroll
          for (int cp = c; cp < CA; ++cp) {
            const double t = __ldg(tau + (row + (cp - c)) * Mk + k);
            const bool ec = !(l_of_c(c) & 1), ecp = !(l_of_c(cp) & 1);
            q[c] = fma(fft_sign(set, ec, ecp) * t, sv[cp][tid], q[c]);
            if (cp != c) q[cp] = fma(fft_sign(set, ecp, ec) * t, vc, q[cp]);
          }
        }
#pragma unroll
        for (int c = 0; c < CA; ++c) {
          const bool ev = !(l_of_c(c) & 1);
          Ohd[2 * ((size_t)(b * CA + c) * Mk + k) + (((set == 0) == ev) ? 0 : 1)] = q[c];
        }
      }
    }
  }
}

// any order: coefficients indexed at run time, table entries read once per output coefficient
__global__ void k_fft_product(const double* tau, const double2* Wh, double2* Oh, int C, int Cact, int nb,
                              size_t Mk) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Mk) return;
  for (int b = 0; b < nb; ++b)
    for (int c = 0; c < Cact; ++c) {
      const bool ec = !(l_of_c(c) & 1);
      double ox = 0.0, oy = 0.0;
      for (int cp = 0; cp < Cact; ++cp) {
        const int lo = min(c, cp), hi = max(c, cp);
        const double t = tau[((size_t)lo * C - (size_t)lo * (lo - 1) / 2 + (hi - lo)) * Mk + k];
        const double2 w = Wh[(size_t)(b * Cact + cp) * Mk + k];
        if (ec == !(l_of_c(cp) & 1)) {  // real spectrum
          ox = fma(t, w.x, ox);
          oy = fma(t, w.y, oy);
        } else {  // i tau
          ox = fma(-t, w.y, ox);
          oy = fma(t, w.x, oy);
        }
      }
      Oh[(size_t)(b * Cact + c) * Mk + k] = make_double2(ox, oy);
    }
}

// The FIM model snaps directions to its SH table, which breaks the parity of T_cc'; its table keeps
// complex spectra and this product reads them directly.
__global__ void k_fft_product_cplx(const double2* That, const double2* Wh, double2* Oh, int C, int Cact, int nb,
                                   size_t Mk) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Mk) return;
  for (int b = 0; b < nb; ++b)
    for (int c = 0; c < Cact; ++c) {
      double ox = 0.0, oy = 0.0;
      for (int cp = 0; cp < Cact; ++cp) {
        const int lo = min(c, cp), hi = max(c, cp);
        const double2 t = That[((size_t)lo * C - (size_t)lo * (lo - 1) / 2 + (hi - lo)) * Mk + k];
        const double2 w = Wh[(size_t)(b * Cact + cp) * Mk + k];
        ox = fma(t.x, w.x, fma(-t.y, w.y, ox));
        oy = fma(t.x, w.y, fma(t.y, w.x, oy));
      }
      Oh[(size_t)(b * Cact + c) * Mk + k] = make_double2(ox, oy);
    }
}

// tau[p][k] = Re or Im of the table spectrum of pair p (by the parity of l + l')
__global__ void k_fft_extract(const double2* spec, double* tau, int p0, int np, int C, size_t Mk) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)np * Mk) return;
  const int q = (int)(t / Mk);
  int p = p0 + q, c = 0;
  while (p >= C - c) {  // row c of the upper triangle holds C - c pairs
    p -= C - c;
    ++c;
  }
  const int cp = c + p;
  const double2 v = spec[t];
  tau[(size_t)p0 * Mk + t] = ((l_of_c(c) + l_of_c(cp)) & 1) ? v.y : v.x;
}

// padded result fields -> split-K partial layout [N][nb][Cfull] (one split), scaled by 1/M
__global__ void k_fft_crop(const double* F, int Cfull, int Cact, int nb, FftTabArgs a, double* part, size_t M) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long N = (long long)a.nx * a.ny * a.nz;
  if (t >= N * nb * Cact) return;
  const int c = (int)(t % Cact);
  const int b = (int)((t / Cact) % nb);
  const long long r = t / ((long long)Cact * nb);
  const int x = (int)(r % a.nx), y = (int)((r / a.nx) % a.ny), z = (int)(r / ((long long)a.nx * a.ny));
  part[(size_t)r * nb * Cfull + (size_t)b * Cfull + c] =
      F[(size_t)(b * Cact + c) * M + ((size_t)z * a.My + y) * a.Mx + x] / (double)M;
}


cudaError_t rte_launch_fft_table(const FftTabArgs& a, int L, int table, double* T, size_t M, cudaStream_t st) {
  const unsigned blocks = (unsigned)((M + 127) / 128);
  switch (L) {
#define RTE_FFT_TAB(LL)                                          \
  case LL:                                                       \
    if (table)                                                   \
      k_fft_table<LL, true><<<blocks, 128, 0, st>>>(a, T, M);    \
    else                                                         \
      k_fft_table<LL, false><<<blocks, 128, 0, st>>>(a, T, M);   \
    break;
    RTE_FFT_TAB(0) RTE_FFT_TAB(1) RTE_FFT_TAB(2) RTE_FFT_TAB(3) RTE_FFT_TAB(4) RTE_FFT_TAB(5) RTE_FFT_TAB(6)
    RTE_FFT_TAB(7)
#undef RTE_FFT_TAB
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t rte_launch_fft_pad(const double* W, int vstride, int Cfull, int Cact, int nb, const FftTabArgs& a, double* F,
                               size_t M, cudaStream_t st) {
  const long long n = (long long)a.nx * a.ny * a.nz * nb * Cact;
  k_fft_pad<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(W, vstride, Cfull, Cact, nb, a, F, M);
  return cudaGetLastError();
}

cudaError_t rte_launch_fft_extract(const void* spec, double* tau, int p0, int np, int C, size_t Mk, cudaStream_t st) {
  const size_t n = (size_t)np * Mk;
  k_fft_extract<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const double2*)spec, tau, p0, np, C, Mk);
  return cudaGetLastError();
}

cudaError_t rte_launch_fft_product(const void* That, const void* Wh, void* Oh, int C, int Cact, int nb, size_t Mk,
                                   int complex_table, cudaStream_t st) {
  const unsigned blocks = (unsigned)((Mk + 127) / 128);
  if (complex_table) {
    k_fft_product_cplx<<<blocks, 128, 0, st>>>((const double2*)That, (const double2*)Wh, (double2*)Oh, C, Cact, nb, Mk);
    return cudaGetLastError();
  }
  const double* T = (const double*)That;
  const double2* W = (const double2*)Wh;
  double2* O = (double2*)Oh;
  const unsigned blocks2 = (unsigned)((2 * Mk + 127) / 128);  // one thread per frequency and set
  switch (Cact) {
    case 1: k_fft_product_reg<0><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    case 4: k_fft_product_reg<1><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    case 9: k_fft_product_reg<2><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    case 16: k_fft_product_reg<3><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    case 25: k_fft_product_reg<4><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    case 36: k_fft_product_reg<5><<<blocks2, 128, 0, st>>>(T, W, O, C, nb, Mk); break;
    default: k_fft_product<<<blocks, 128, 0, st>>>(T, W, O, C, Cact, nb, Mk);
  }
  return cudaGetLastError();
}

cudaError_t rte_launch_fft_crop(const double* F, int Cfull, int Cact, int nb, const FftTabArgs& a, double* part,
                                size_t M, cudaStream_t st) {
  const long long n = (long long)a.nx * a.ny * a.nz * nb * Cact;
  k_fft_crop<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, Cfull, Cact, nb, a, part, M);
  return cudaGetLastError();
}

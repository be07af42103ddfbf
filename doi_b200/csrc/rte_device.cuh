// Device code shared by the kernel files: packed FP32 arithmetic, compile-time SH normalisations, the
// reference's direction table, bulk copies and their bounded waits.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "rte_internal.h"

// Packed FP32 pairs (sm_100 f32x2 arithmetic): two FP32 FMAs per instruction.
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
  f2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
  f2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Compile-time copies of the SH recurrence coefficients (the same formulas as the host tables in rte_host.cpp).
struct ShConstTab {
  double A[64], B[64], Q0[RTE_MAX_L + 1];
};
constexpr double c_sqrt(double x) {
  double r = x > 1.0 ? x : 1.0;
  for (int i = 0; i < 80; ++i) r = 0.5 * (r + x / r);
  return r;
}
constexpr double c_knorm(int l, int m) {
  double f = 1.0;
  for (int i = l - m + 1; i <= l + m; ++i) f *= (double)i;
  const double k = c_sqrt((2.0 * l + 1.0) / (4.0 * 3.14159265358979323846) / f);
  return m > 0 ? k * c_sqrt(2.0) : k;
}
constexpr ShConstTab make_sh_const() {
  ShConstTab t{};
  for (int m = 0; m <= RTE_MAX_L; ++m) {
    double dfact = 1.0;
    for (int i = 2 * m - 1; i > 0; i -= 2) dfact *= (double)i;
    t.Q0[m] = c_knorm(m, m) * ((m & 1) ? -1.0 : 1.0) * dfact;
    for (int l = m + 1; l <= RTE_MAX_L; ++l) {
      const int id = l * (l + 1) / 2 + m;
      t.A[id] = c_knorm(l, m) * (2.0 * l - 1.0) / ((double)(l - m) * c_knorm(l - 1, m));
      t.B[id] = (l - 2 >= m) ? c_knorm(l, m) * (double)(l + m - 1) / ((double)(l - m) * c_knorm(l - 2, m)) : 0.0;
    }
  }
  return t;
}

// Monic form of the SH recurrence.  With q_l^m = s_lm u_l^m, s_mm = Q0[m] and s_lm = A_lm s_{l-1,m}, the
// polynomials u satisfy u_l = z u_{l-1} - beta_lm u_{l-2} (beta_lm = B_lm s_{l-2,m} / s_lm), so R_c = N_c U_c with
// U_{l,+-m} = u_l^m Re/Im((x+iy)^m) and N_c = s_lm.  The column kernels work with U: the factors N_c are applied
// once per source row (the rows hold N_c W_c) and once per destination.
struct MonicTab {
  double beta[64];  // index l*(l+1)/2 + m
  double N[64];     // index l*l + l + m
};
constexpr MonicTab make_monic() {
  MonicTab t{};
  const ShConstTab q = make_sh_const();
  for (int m = 0; m <= RTE_MAX_L; ++m) {
    double s[RTE_MAX_L + 1] = {};
    s[m] = q.Q0[m];
    for (int l = m + 1; l <= RTE_MAX_L; ++l) s[l] = q.A[l * (l + 1) / 2 + m] * s[l - 1];
    for (int l = m; l <= RTE_MAX_L; ++l) {
      if (l >= m + 2) t.beta[l * (l + 1) / 2 + m] = q.B[l * (l + 1) / 2 + m] * s[l - 2] / s[l];
      t.N[l * l + l + m] = s[l];
      t.N[l * l + l - m] = s[l];
    }
  }
  return t;
}
__device__ constexpr MonicTab kMonic = make_monic();

// Direction snapped to the reference's 100x100 SH table cell (FisherInfo_IO/src/defines.h:53-56
// and kernels.cu:326-333: theta = acos(dz/dist), phi = atan2(dy,dx) NOT wrapped to [0,2pi), so a
// negative phi index reads the previous theta row of the flat table).
__device__ __forceinline__ void table_direction(double ddx, double ddy, double ddz, double dist, double& ux,
                                                double& uy, double& uz) {
  double theta = acos(ddz / dist);
  double phi = atan2(ddy, ddx);
  int ti = (int)rintf((float)((100 - 1) * (theta) / (M_PI)));
  int pj = (int)rintf((float)((100 - 1) * (phi) / (2 * M_PI)));
  int off = ti * 100 + pj;
  if (off < 0) off = 0;
  int tq = off / 100, pq = off - tq * 100;
  double th = (tq * M_PI) / (100 - 1);
  double ph = (pq * 2.0 * M_PI) / (100 - 1);
  double st, ct, sp, cp;
  sincos(th, &st, &ct);
  sincos(ph, &sp, &cp);
  ux = st * cp;
  uy = st * sp;
  uz = ct;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// bounded wait on an mbarrier phase; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Tensor memory as a per-thread accumulator store: 128 lanes x 512 columns of 32 bits per SM; warp w of a CTA owns
// lanes 32 (w % 4) .. + 31, so each thread of a 128-thread CTA has the CTA's allocated columns of its own lane.
// All of these are .sync.aligned: a warp executes them converged, with a __syncwarp() behind whatever may have split it.
template <int N>
__device__ __forceinline__ void tmem_ld_x(uint32_t addr, uint32_t* v);
template <int N>
__device__ __forceinline__ void tmem_st_x(uint32_t addr, const uint32_t* v);
template <>
__device__ __forceinline__ void tmem_ld_x<1>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v[0]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<1>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr), "r"(v[0]));
}
template <>
__device__ __forceinline__ void tmem_ld_x<2>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<2>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v[0]), "r"(v[1]));
}
template <>
__device__ __forceinline__ void tmem_ld_x<4>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<4>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
}
template <>
__device__ __forceinline__ void tmem_ld_x<8>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<8>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
}
template <>
__device__ __forceinline__ void tmem_ld_x<16>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<16>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]));
}
template <>
__device__ __forceinline__ void tmem_ld_x<32>(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]) : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_st_x<32>(uint32_t addr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]));
}
// N consecutive columns; the registers of a load are valid after tmem_wait_ld
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t* v) {
  constexpr int P = N >= 32 ? 32 : (N >= 16 ? 16 : (N >= 8 ? 8 : (N >= 4 ? 4 : (N >= 2 ? 2 : 1))));
  tmem_ld_x<P>(addr, v);
  if constexpr (N > P) tmem_ld<N - P>(addr + P, v + P);
}
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t* v) {
  constexpr int P = N >= 32 ? 32 : (N >= 16 ? 16 : (N >= 8 ? 8 : (N >= 4 ? 4 : (N >= 2 ? 2 : 1))));
  tmem_st_x<P>(addr, v);
  if constexpr (N > P) tmem_st<N - P>(addr + P, v + P);
}
// The loaded registers pass through an empty statement behind the wait, so that no arithmetic on them, which depends on
// registers alone, is scheduled ahead of it.
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t* v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < N; ++q) asm volatile("" : "+r"(v[q]));
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// one warp allocates (address to shared memory) and frees
__device__ __forceinline__ void tmem_alloc(uint32_t* smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

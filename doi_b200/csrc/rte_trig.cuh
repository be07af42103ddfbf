// Real spherical harmonics of order <= L on one meridian as trigonometric polynomials of the polar angle: the
// contraction of coefficient rows onto a meridian and its transpose (rte_column.cu, rte_backproject.cu).
#pragma once
#include "rte_device.cuh"

// a[l][m][k]: U_lm = sum_k a cos(k theta) (m even) or a sin(k theta) (m odd), U the monic associated
// Legendre functions sin^m u_l^m of the recurrence u_l = cos u_{l-1} - beta u_{l-2}
struct TrigTab {
  double a[RTE_MAX_L + 1][RTE_MAX_L + 1][RTE_MAX_L + 1];
};
constexpr TrigTab make_trig() {
  TrigTab t{};
  const MonicTab mo = make_monic();
  double mm[RTE_MAX_L + 2] = {};  // U_mm = sin^m
  mm[0] = 1.0;
  for (int m = 0; m <= RTE_MAX_L; ++m) {
    if (m > 0) {
      double n[RTE_MAX_L + 2] = {};
      for (int k = 0; k < RTE_MAX_L; ++k) {
        if ((m - 1) % 2 == 0) {  // cos k sin = (sin(k+1) - sin(k-1)) / 2
          n[k + 1] += 0.5 * mm[k];
          if (k == 0)
            n[1] += 0.5 * mm[k];  // -sin(-1) = sin 1
          else if (k > 1)
            n[k - 1] -= 0.5 * mm[k];
        } else if (k > 0) {  // sin k sin = (cos(k-1) - cos(k+1)) / 2
          n[k - 1] += 0.5 * mm[k];
          n[k + 1] -= 0.5 * mm[k];
        }
      }
      for (int k = 0; k <= RTE_MAX_L + 1; ++k) mm[k] = n[k];
    }
    double p[RTE_MAX_L + 2] = {}, q[RTE_MAX_L + 2] = {};  // l - 1, l - 2
    for (int k = 0; k <= RTE_MAX_L; ++k) q[k] = 0.0, p[k] = mm[k];
    for (int k = 0; k <= RTE_MAX_L; ++k) t.a[m][m][k] = mm[k];
    for (int l = m + 1; l <= RTE_MAX_L; ++l) {
      double n[RTE_MAX_L + 2] = {};
      for (int k = 0; k < l; ++k) {  // times cos
        if (m % 2 == 0) {
          n[k + 1] += 0.5 * p[k];
          n[k == 0 ? 1 : k - 1] += 0.5 * p[k];
        } else if (k > 0) {
          n[k + 1] += 0.5 * p[k];
          if (k > 1) n[k - 1] += 0.5 * p[k];
        }
      }
      const double b = l >= m + 2 ? mo.beta[l * (l + 1) / 2 + m] : 0.0;
      for (int k = 0; k <= RTE_MAX_L; ++k) {
        n[k] -= b * q[k];
        q[k] = p[k];
        p[k] = n[k];
        t.a[l][m][k] = n[k];
      }
    }
  }
  return t;
}
__device__ constexpr TrigTab kTrig = make_trig();

__host__ __device__ constexpr int up4(int n) { return (n + 3) / 4 * 4; }

// numbers per (source, destination column, right-hand side): (cos k, sin k) pairs k = 1..L, then (k = 0, 0)
template <int L>
__host__ __device__ constexpr int nb_row() {
  return up4(2 * L + 2);
}

// The pairs p_k = (cos k theta, sin k theta) follow p_{k+2} = 2 cos 2theta p_k - p_{k-2} from p_{-1}, p_0, p_1, p_2.
template <int L, typename T>
__device__ __forceinline__ void trig_pairs(T c1, T s1, T c2, T s2, T* c, T* s) {
  if constexpr (L >= 1) c[0] = c1, s[0] = s1;
  if constexpr (L >= 2) c[1] = c2, s[1] = s2;
  const T t = c2 + c2;
#pragma unroll
  for (int k = 3; k <= L; ++k) {
    if (k == 3) {
      c[2] = fma(t, c1, -c1);
      s[2] = fma(t, s1, s1);
    } else if (k == 4) {
      c[3] = fma(t, c2, T(-1));
      s[3] = t * s2;
    } else {
      c[k - 1] = fma(t, c[k - 3], -c[k >= 5 ? k - 5 : 0]);
      s[k - 1] = fma(t, s[k - 3], -s[k >= 5 ? k - 5 : 0]);
    }
  }
}

// row of one source -> its 2L+1 numbers for a column at azimuth (cm, sm)
template <int L, typename T>
__device__ __forceinline__ void contract_row(const T* w, const T* __restrict__ az, T* b) {
#pragma unroll
  for (int k = 0; k < nb_row<L>(); ++k) b[k] = T(0);
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    const T cm = m > 0 ? az[2 * (m > 0 ? m : 1) - 2] : T(1), sm = m > 0 ? az[2 * (m > 0 ? m : 1) - 1] : T(0);
#pragma unroll
    for (int l = m; l <= L; ++l) {
      const T z = m > 0 ? fma(cm, w[l * l + l + m], sm * w[l * l + l - m]) : w[l * l + l];
#pragma unroll
      for (int k = l & 1; k <= l; k += 2) {
        if (m % 2 == 1 && k == 0) continue;
        const int q = k == 0 ? 2 * L : (2 * k - 2 + (m & 1));
        b[q] = fma((T)kTrig.a[l][m][k], z, b[q]);
      }
    }
  }
}

// sums of one source column -> destination coefficients (adds to out)
template <int L, typename T>
__device__ __forceinline__ void expand_row(const T* g, const T* __restrict__ az, T* out) {
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    const T cm = m > 0 ? az[2 * (m > 0 ? m : 1) - 2] : T(1), sm = m > 0 ? az[2 * (m > 0 ? m : 1) - 1] : T(0);
#pragma unroll
    for (int l = m; l <= L; ++l) {
      T z = T(0);
#pragma unroll
      for (int k = l & 1; k <= l; k += 2) {
        if (m % 2 == 1 && k == 0) continue;
        const int q = k == 0 ? 2 * L : (2 * k - 2 + (m & 1));
        z = fma((T)kTrig.a[l][m][k], g[q], z);
      }
      if (m == 0) {
        out[l * l + l] += z;
      } else {
        out[l * l + l + m] = fma(cm, z, out[l * l + l + m]);
        out[l * l + l - m] = fma(sm, z, out[l * l + l - m]);
      }
    }
  }
}

// Per-edge basis functions evaluated in registers: real spherical harmonics Y_lm(d/|d|) and the
// tanh-warped Chebyshev radial basis with its cutoff envelope.
//
// Real Y_lm.  Same convention as the reference engine (interfaces/lammps/ML-SUS2/sus2_sl_kernel.cpp:
// 12-42: orthonormal, Condon-Shortley phase folded so that Y_l,+m ~ +Re (x+iy)^m, index
// h = l*l + l + m).  Formulated here on the unit vector u = d/r:
//     Y_l,0  = f_l0(u_z)
//     Y_l,+m = f_lm(u_z) Re (u_x + i u_y)^m,   Y_l,-m = f_lm(u_z) Im (u_x + i u_y)^m
// where f_lm = N_lm Pi_lm (times sqrt(2) for m > 0), N_lm = sqrt((2l+1)/(4 pi) (l-m)!/(l+m)!),
// Pi_mm = (2m-1)!! and Pi_lm = ((2l-1) u_z Pi_l-1,m - (l+m-1) Pi_l-2,m) / (l-m) (the
// associated-Legendre recurrence with |u| = 1 substituted).  The normalisation is folded into the
// coefficients at compile time; up to l = m + 3 f_lm is its polynomial in u_z, above it the
// recurrence.  Sums over l come before the products with (u_x + i u_y)^m.  Every pass evaluates
// these per edge and is bound by its instructions (FP64: by the FP64 pipe); terms times constant
// zeros and ones, which the compiler has to keep, are left out (with the virial's halving sums: adjoint
// of Static L3/K4/O2, 32,768 atoms, 138.5 -> 129.1 us; gate reverse of Effect L4/K8/R2/O3, 8,000
// atoms, 112.5 -> 104.6 us).  The gradient with respect to d
// only needs tangential derivatives, so any smooth extension Yhat(u) off the sphere gives
//     dY/dd = (1/r) (I - u u^T) grad_u Yhat(u),
// which the reverse and tangent helpers below use with the polynomial extension above.
//
// Radial basis RBChebyshev_sss (src/radial_basis.cpp:1259, sus2_sl_radial_math.cpp:468-500,
// 1543-1595): xi = tanh(s (r - sigma) / 2), T_0 = 1, T_1 = xi, T_b = 2 xi T_b-1 - T_b-2, times
// scaling * f_c(r) with the legacy envelope f_c = (r - r_c)^2 or the polynomial envelope
// (sus2_sl_radial_math.cpp:256-294).  With two cutoffs the l = 0 functions use max_dist and the
// l > 0 functions use angular_max_dist (RB_CalcForCutoff, sus2_sl_radial_math.cpp:296-336).
#pragma once
#include <cmath>
#include <type_traits>
#include <utility>

#include "device_common.cuh"

namespace sus2g {

__host__ __device__ constexpr int sh_index(int l, int m) { return l * l + l + m; }

// sqrt by Newton's method (from above, until it stops falling), for constants only
__host__ __device__ constexpr double const_sqrt(double x) {
  double r = x > 1.0 ? x : 1.0;
  for (double n = 0.5 * (r + x / r); n < r; n = 0.5 * (r + x / r)) r = n;
  return r;
}
// N_lm, times sqrt(2) for m > 0, times (2m-1)!!
__host__ __device__ constexpr double sph_norm(int l, int m) {
  double ratio = 1.0, dfact = 1.0;
  for (int a = l - m + 1; a <= l + m; ++a) ratio /= a;
  for (int a = 3; a <= 2 * m - 1; a += 2) dfact *= a;
  return const_sqrt((2 * l + 1) * ratio / (4 * 3.14159265358979323846) * (m ? 2.0 : 1.0)) * dfact;
}

// f(A), f(A + 1) .. f(N - 1) with the index as a compile-time constant.
template <int A, int N, typename Fn>
__device__ __forceinline__ void unroll(Fn&& fn) {
  if constexpr (A < N) {
    fn(std::integral_constant<int, A>{});
    unroll<A + 1, N>(fn);
  }
}

// f_lm(z) for l = m .. L into f[l - m], and df_lm/dz into d[l - m] (DERIV).
template <int L, int m, bool DERIV, typename T>
__device__ __forceinline__ void legendre_column(T z, T z2, T* f, T* d) {
  unroll<m, L + 1>([&](auto lc) {
    constexpr int l = decltype(lc)::value, q = l - m;
    constexpr double n = sph_norm(l, m);
    if constexpr (q == 0) {
      f[0] = T(n);
      if (DERIV) d[0] = T(0);
    } else if constexpr (q == 1) {
      constexpr double c = n * (2 * m + 1);
      f[1] = T(c) * z;
      if (DERIV) d[1] = T(c);
    } else if constexpr (q == 2) {
      constexpr double c = n * (2 * m + 1) / 2, a = c * (2 * m + 3), a2 = 2 * a;
      f[2] = T(a) * z2 - T(c);
      if (DERIV) d[2] = T(a2) * z;
    } else if constexpr (q == 3) {
      constexpr double b = n * (2 * m + 1) * (2 * m + 3) / 6, a = b * (2 * m + 5), a3 = 3 * a, b3 = 3 * b;
      f[3] = z * (T(a) * z2 - T(b3));
      if (DERIV) d[3] = T(a3) * z2 - T(b3);
    } else {
      constexpr double a = n / sph_norm(l - 1, m) * (2 * l - 1) / q, b = n / sph_norm(l - 2, m) * (l + m - 1) / q;
      f[q] = T(a) * z * f[q - 1] - T(b) * f[q - 2];
      if (DERIV) d[q] = T(a) * (z * d[q - 1] + f[q - 1]) - T(b) * d[q - 2];
    }
  });
}

// (u_x + i u_y)^m for m = 0 .. L
template <int L, typename T>
__device__ __forceinline__ void azimuth_powers(T ux, T uy, T* Cm, T* Sm) {
  Cm[0] = T(1); Sm[0] = T(0);
  if (L >= 1) { Cm[1] = ux; Sm[1] = uy; }
#pragma unroll
  for (int m = 2; m <= L; ++m) {
    Cm[m] = ux * Cm[m - 1] - uy * Sm[m - 1];
    Sm[m] = ux * Sm[m - 1] + uy * Cm[m - 1];
  }
}

// Values Y[h] for h < (L+1)^2 at unit vector (ux, uy, uz).
template <int L, typename T>
__device__ __forceinline__ void sph_values(T ux, T uy, T uz, T* Y) {
  T Cm[L + 1], Sm[L + 1];
  azimuth_powers<L>(ux, uy, Cm, Sm);
  const T z2 = uz * uz;
  unroll<0, L + 1>([&](auto mc) {
    constexpr int m = decltype(mc)::value;
    T f[L + 1 - m];
    legendre_column<L, m, false, T>(uz, z2, f, nullptr);
#pragma unroll
    for (int l = m; l <= L; ++l) {
      if (m == 0) {
        Y[sh_index(l, 0)] = f[l];
      } else {
        Y[sh_index(l, m)] = f[l - m] * Cm[m];
        Y[sh_index(l, -m)] = f[l - m] * Sm[m];
      }
    }
  });
}

// grad_u of sum_h P[h] Yhat_h(u) (polynomial extension), accumulated into (gx, gy, gz).
template <int L, typename T>
__device__ __forceinline__ void sph_grad_dot(T ux, T uy, T uz, const T* P, T& gx, T& gy, T& gz) {
  T Cm[L + 1], Sm[L + 1];
  azimuth_powers<L>(ux, uy, Cm, Sm);
  const T z2 = uz * uz;
  unroll<0, L + 1>([&](auto mc) {
    constexpr int m = decltype(mc)::value;
    T f[L + 1 - m], d[L + 1 - m];
    legendre_column<L, m, true, T>(uz, z2, f, d);
    if constexpr (m == 0) {
#pragma unroll
      for (int l = 1; l <= L; ++l) gz += P[sh_index(l, 0)] * d[l];
    } else {
      // sums over l, then d/dux (C_m, S_m) = m (C_m-1, S_m-1), d/duy (C_m, S_m) = m (-S_m-1, C_m-1)
      T fc = f[0] * P[sh_index(m, m)], fs = f[0] * P[sh_index(m, -m)], dc = T(0), ds = T(0);
#pragma unroll
      for (int l = m + 1; l <= L; ++l) {
        fc += f[l - m] * P[sh_index(l, m)];
        fs += f[l - m] * P[sh_index(l, -m)];
        if (l == m + 1) {
          dc = d[1] * P[sh_index(l, m)];
          ds = d[1] * P[sh_index(l, -m)];
        } else {
          dc += d[l - m] * P[sh_index(l, m)];
          ds += d[l - m] * P[sh_index(l, -m)];
        }
      }
      if constexpr (m == 1) {
        gx += fc;
        gy += fs;
      } else {
        fc *= T(m);
        fs *= T(m);
        gx += fc * Cm[m - 1] + fs * Sm[m - 1];
        gy += fs * Cm[m - 1] - fc * Sm[m - 1];
      }
      if constexpr (m < L) gz += dc * Cm[m] + ds * Sm[m];
    }
  });
}

// Tangent of Yhat along a tangential direction t (already projected, divided by r):
// Ydot[h] = t . grad_u Yhat_h.
template <int L, typename T>
__device__ __forceinline__ void sph_tangent(T ux, T uy, T uz, T tx, T ty, T tz, T* Ydot) {
  T Cm[L + 1], Sm[L + 1];
  azimuth_powers<L>(ux, uy, Cm, Sm);
  const T z2 = uz * uz;
  unroll<0, L + 1>([&](auto mc) {
    constexpr int m = decltype(mc)::value;
    T f[L + 1 - m], d[L + 1 - m];
    legendre_column<L, m, true, T>(uz, z2, f, d);
    if constexpr (m == 0) {
      Ydot[0] = T(0);
#pragma unroll
      for (int l = 1; l <= L; ++l) Ydot[sh_index(l, 0)] = d[l] * tz;
    } else {
      // the tangents of C_m and S_m, and tz C_m, tz S_m
      const T ct = m == 1 ? tx : T(m) * (Cm[m - 1] * tx - Sm[m - 1] * ty);
      const T st = m == 1 ? ty : T(m) * (Sm[m - 1] * tx + Cm[m - 1] * ty);
      const T cz = Cm[m] * tz, sz = Sm[m] * tz;
      Ydot[sh_index(m, m)] = f[0] * ct;
      Ydot[sh_index(m, -m)] = f[0] * st;
#pragma unroll
      for (int l = m + 1; l <= L; ++l) {
        Ydot[sh_index(l, m)] = f[l - m] * ct + d[l - m] * cz;
        Ydot[sh_index(l, -m)] = f[l - m] * st + d[l - m] * sz;
      }
    }
  });
}

// Warp variable and its derivatives for the parameter gradient: xi = tanh(s (r - sigma) / 2).
template <typename T>
struct WarpVar {
  T xi, xr, xs, xg, xrs, xrg;  // xi, d/dr, d/ds, d/dsigma, d2/dr ds, d2/dr dsigma
};

template <typename T>
__device__ __forceinline__ WarpVar<T> warp_var(T r, T slope, T shift) {
  WarpVar<T> w;
  w.xi = tanh(slope * (r - shift) * T(0.5));
  const T e = T(1) - w.xi * w.xi;
  w.xr = e * slope * T(0.5);
  w.xs = e * (r - shift) * T(0.5);
  w.xg = -e * slope * T(0.5);
  w.xrs = e * T(0.5) - w.xi * w.xs * slope;
  w.xrg = -w.xi * w.xg * slope;
  return w;
}

// Chebyshev T_b(xi) with its first and second derivatives in xi, b < B <= NBM <= kMaxB.
template <typename T, int NBM = kMaxB>
__device__ __forceinline__ void cheb_full(T xi, int B, T* Tv, T* D, T* DD) {
  Tv[0] = T(1); D[0] = T(0); DD[0] = T(0);
  Tv[1] = xi; D[1] = T(1); DD[1] = T(0);
#pragma unroll
  for (int b = 2; b < NBM; ++b) {
    if (b < B) {
      Tv[b] = T(2) * xi * Tv[b - 1] - Tv[b - 2];
      D[b] = T(2) * Tv[b - 1] + T(2) * xi * D[b - 1] - D[b - 2];
      DD[b] = T(4) * D[b - 1] + T(2) * xi * DD[b - 1] - DD[b - 2];
    }
  }
}

// Cutoff envelope f_c and its r-derivative (CalcRadialCutoff, sus2_sl_radial_math.cpp:256-294).
template <typename T>
__device__ __forceinline__ void envelope(T r, T rc, int poly, int p, T& f, T& fd) {
  if (r >= rc) { f = T(0); fd = T(0); return; }
  if (!poly) {
    const T dr = r - rc;
    f = dr * dr;
    fd = T(2) * dr;
    return;
  }
  const T x = r / rc, omx = T(1) - x;
  T poly_v = T(0);
  for (int k = p - 1; k >= 0; --k) poly_v = poly_v * x + T(0.5) * T((k + 1) * (k + 2));
  f = omx * omx * omx * poly_v;
  T xp = T(1);
  for (int k = 0; k < p - 1; ++k) xp *= x;
  const T pf = T(p);
  fd = T(-0.5) * pf * (pf + T(1)) * (pf + T(2)) * xp * omx * omx / rc;
}

}  // namespace sus2g

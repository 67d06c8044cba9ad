// ytf_bessel.cuh -- Bessel functions J_0, J_1, J_2 of a complex argument (device), for the
// synthesis on a deformed kρ contour (kρ ρ complex, close to the real axis for most radii). Published
// methods by range:
//   0 <= Re z < 25, |Im z| <= 0.4 : the Taylor rows of J_0 about i + 1/2 (ytf_bessel_tab.cuh) at the
//                   complex distance d, |d| <= 0.65: one complex Horner pass for the value and the
//                   derivative -J_1, |error| < 1e-15; J_1 below |z| = 1 from its series, for its relative
//                   accuracy;
//   |z| >= 25     : the Hankel asymptotic expansion J_n(z) = √(2/(πz)) (P cos χ - Q sin χ),
//                   χ = z - nπ/2 - π/4 (A&S 9.2.5, 9.2.9-10), P and Q as polynomials in 1/z² up to
//                   the 19th term (the next is below 1e-17 at |z| = 25), both orders from one phase;
//   |z| <= 8      : the power series J_n(z) = (z/2)^n Σ_m (-z²/4)^m / (m! (m+n)!)
//                   (A&S 9.1.10); the largest term is ~1e2, so ~1e-14 absolute accuracy;
//   8 < |z| < 25  : Miller's backward recurrence J_{k-1} = (2k/z) J_k - J_{k+1} from an order
//                   N = |z| + 32 with the normalisation J_0 + 2 Σ_{k≥1} J_{2k} = 1 (A&S 9.1.27,
//                   9.1.46), valid for complex z.
// J_2 from the recurrence 2J_1/z - J_0 above |z| = 1, from its series below. Principal
// branches (Re z > 0 on the contour). Bound by FP64 issue: 256 radii x 4096 contour nodes with
// the slice maxima took 98 + 40 us with series, Miller and a 24-term complex loop per order and a pass
// over the tables for the maxima; 31 us with the Taylor rows, the polynomials and the maxima per warp.
#pragma once
#include "ytf_bessel_tab.cuh"
#include "ytf_complex.cuh"

namespace ytf {

// (z/2)^n Σ_m (-z²/4)^m / (m! (m+n)!), n = 0, 1, 2
__device__ inline cd bessel_series(int n, cd z) {
  const cd h = z * 0.5;
  const cd q = -(h * h);
  cd t{1.0, 0.0};
  double f = 1.0;
  for (int i = 1; i <= n; ++i) f *= i;
  t = t * (1.0 / f);
  cd s = t;
  for (int m = 1; m < 60; ++m) {
    t = t * q * (1.0 / ((double)m * (double)(m + n)));
    s += t;
    if (norm2(t) < 1e-36 * norm2(s)) break;
  }
  cd p{1.0, 0.0};
  for (int i = 0; i < n; ++i) p = p * h;
  return s * p;
}

// N! (2/z)^N J_N(z) = Σ_m (-h2)^m N! / (m! (m + N)!), h2 = z²/4, below |z| = 1 (A&S 9.1.10; 9 terms, the
// first left out under 1e-17), of a real or complex argument
template <int N>
__device__ __forceinline__ double bessel_series_unit(double h2) {
  double s = 1.0;
#pragma unroll
  for (int m = 8; m >= 1; --m) s = fma(-(h2 * (1.0 / (m * (m + N)))), s, 1.0);
  return s;
}
template <int N>
__device__ __forceinline__ cd bessel_series_unit(cd h2) {
  cd s{1.0, 0.0};
#pragma unroll
  for (int m = 8; m >= 1; --m) {
    s = (h2 * s) * (-1.0 / (m * (m + N)));
    s.x += 1.0;
  }
  return s;
}

// Hankel's coefficients a_k(n) = Π_{j<=k} (4n² - (2j - 1)²) / (k! 8^k)
struct HankelCoef {
  double a[2][20];
};
__host__ __device__ constexpr HankelCoef hankel_coef() {
  HankelCoef h{};
  for (int n = 0; n < 2; ++n) {
    h.a[n][0] = 1.0;
    for (int k = 1; k < 20; ++k) h.a[n][k] = h.a[n][k - 1] * (4.0 * n * n - (2.0 * k - 1) * (2.0 * k - 1)) / (8.0 * k);
  }
  return h;
}
// Σ_{k = first, first + 2, ... <= 19} ± a_k w^{(k - first) / 2}, signs alternating from +
template <int N, int FIRST>
__device__ __forceinline__ cd hankel_sum(cd w) {
  constexpr HankelCoef h = hankel_coef();
  cd s{(9 % 2 ? -1.0 : 1.0) * h.a[N][FIRST + 18], 0.0};
#pragma unroll
  for (int i = 8; i >= 0; --i) {
    s = s * w;
    s.x += (i % 2 ? -1.0 : 1.0) * h.a[N][FIRST + 2 * i];
  }
  return s;
}

template <int N, int FIRST>
__device__ __forceinline__ double hankel_sum(double w) {
  constexpr HankelCoef h = hankel_coef();
  double s = (9 % 2 ? -1.0 : 1.0) * h.a[N][FIRST + 18];
#pragma unroll
  for (int i = 8; i >= 0; --i) s = fma(s, w, (i % 2 ? -1.0 : 1.0) * h.a[N][FIRST + 2 * i]);
  return s;
}

__device__ inline void bessel_j01_c(cd z, cd& J0, cd& J1) {
  if (z.x >= 0.0 && z.x < (double)JTAB_N && fabs(z.y) <= 0.4) {
    const int i = (int)z.x;
    const cd d{z.x - ((double)i + 0.5), z.y};
    const double* c = JTAB + i * JTAB_M;
    cd p{c[JTAB_M - 1], 0.0}, q{0.0, 0.0};
#pragma unroll
    for (int m = JTAB_M - 2; m >= 0; --m) {
      q = q * d + p;
      p = p * d;
      p.x += c[m];
    }
    J0 = p;
    // near 0 the derivative holds J_1 = z/2 to 1e-17 of 1, not of itself
    J1 = norm2(z) < 1.0 ? z * 0.5 * bessel_series_unit<1>(z * z * 0.25) : -q;
    return;
  }
  const double az = cabs(z);
  if (az <= 8.0) {
    J0 = bessel_series(0, z);
    J1 = bessel_series(1, z);
    return;
  }
  if (az < 25.0) {
    const int N = 2 * (((int)az + 32) / 2);  // even start order
    const cd iz = recip(z);
    cd jp1{0.0, 0.0}, jk{1e-200, 0.0};
    cd sum{0.0, 0.0}, j0v{0.0, 0.0}, j1v{0.0, 0.0};
    for (int k = N; k >= 1; --k) {
      const cd jm1 = iz * (2.0 * k) * jk - jp1;  // J_{k-1}
      jp1 = jk;
      jk = jm1;
      const int km1 = k - 1;
      if (km1 > 0 && (km1 % 2) == 0) sum += jk * 2.0;
      if (km1 == 1) j1v = jk;
      if (km1 == 0) j0v = jk;
      if (cabs1(jk) > 1e200) {  // rescale on growth
        jk = jk * 1e-200; jp1 = jp1 * 1e-200; sum = sum * 1e-200; j1v = j1v * 1e-200;
      }
    }
    sum += j0v;
    const cd r = recip(sum);
    J0 = j0v * r;
    J1 = j1v * r;
    return;
  }
  // Hankel asymptotic expansion
  const cd iz = recip(z), w = iz * iz;
  const cd sq = csqrt(iz * (2.0 / 3.14159265358979323846));
  const cd P0 = hankel_sum<0, 0>(w), Q0 = iz * hankel_sum<0, 1>(w);
  const cd P1 = hankel_sum<1, 0>(w), Q1 = iz * hankel_sum<1, 1>(w);
  // cos z and sin z, then χ_0 = z - π/4, χ_1 = χ_0 - π/2
  double sx, cx;
  sincos(z.x, &sx, &cx);
  const double sh = sinh(z.y), ch = fabs(sh) < 1e150 ? sqrt(fma(sh, sh, 1.0)) : fabs(sh);
  const cd cz{cx * ch, -sx * sh}, sz{sx * ch, cx * sh};
  const cd c0 = (cz + sz) * 0.70710678118654752440, s0 = (sz - cz) * 0.70710678118654752440;
  J0 = sq * (P0 * c0 - Q0 * s0);
  J1 = sq * (P1 * s0 + Q1 * c0);
}

__device__ inline void bessel_j012_c(cd z, cd& J0, cd& J1, cd& J2) {
  bessel_j01_c(z, J0, J1);
  if (norm2(z) < 1.0) J2 = bessel_series(2, z);
  else J2 = recip(z) * J1 * 2.0 - J0;
}

}  // namespace ytf

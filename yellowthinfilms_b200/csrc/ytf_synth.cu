// ytf_synth.cu -- synthesis of G(ρ, z, z') from a device transfer cache.
//
// 1D (point source, azimuthally symmetric stack; closed_form_G for CavityTransferCache1D,
// mod_ClosedFormField.jl:435-487): the Jacobi–Anger pixel integral
// (_integrate_pixel_1d, :344-390) is linear in (J0, J1, J2)(kρ), so for every distinct
// radius and z-row it is the contraction
//     R[ρ, col] = Σ_k J_n(k ρ) · C_n[k, col],   n = 0, 1, 2,
// of a Bessel table with per-node coefficients (weighted amplitude × mode field × phase ×
// k). k_coef_sym (5 complex columns per z-row, where TE and TM decouple) or k_coef1d_amp (9) build
// C_n, k_bessel the tables, k_gemm64 does the contractions and k_assemble1d combines orders,
// rotates by the pixel azimuth and writes Julia's (Nx, Ny, Nz, 3, 3) column-major layout.
//
// 2D (any stack; closed_form_G for CavityTransferCache2D, lateral=:direct, :711-753):
// k_strengths_rows forms the 9 strengths per (node, z-row) (_strengths_row!, :616-659) and
// k_lateral64 evaluates G[pix, col] = Σ_n e^{i(kx_n x + ky_n y)} S[col, n] as a complex GEMM
// whose A operand is formed from the x and y phase tables (k_strengths2d and k_lateral: the
// allocation-free entry point's forms of the two).
#include "ytf_complex.cuh"
#include "ytf_kernels.h"
#include "ytf_bessel.cuh"

#include <algorithm>

namespace ytf {

__device__ __forceinline__ cd ldc(const double2* b, long e, long n, long i) {
  double2 v = b[e * n + i];
  return cd{v.x, v.y};
}

// 16-byte asynchronous copy to shared memory, the bytes past `bytes` zero
__device__ __forceinline__ void cp16(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// _phase (mod_ClosedFormField.jl:59-69): clamped exp(i kz z)
__device__ __forceinline__ cd phase_cl(cd kz, double z) {
  double a = -kz.y * z, b = kz.x * z;
  if (!isfinite(a) || !isfinite(b) || a > 700.0 || a < -700.0) return cd{0.0, 0.0};
  return cexp(cd{a, b});
}
// e^{a + i b}, out of line: the exact phases are the rare case of the recurrence over the heights
__device__ __noinline__ cd cexp_call(double a, double b) { return cexp(cd{a, b}); }
__device__ __forceinline__ cd phase_call(cd kz, double z) { return cexp_call(-kz.y * z, kz.x * z); }

__device__ __forceinline__ cd fin0(cd z) { return isfin(z) ? z : cd{0.0, 0.0}; }

// reflected amplitudes of node k (amplitude_at, :175-203) with the term masks
__device__ __forceinline__ void reflected_amp(const SynthParams& p, long k, cd Af[2][3], cd Ab[2][3]) {
  const CacheView& c = p.c;
  for (int m = 0; m < 2; ++m)
    for (int q = 0; q < 3; ++q) { Af[m][q] = cd{0, 0}; Ab[m][q] = cd{0, 0}; }
  if (!(c.valid[k] && c.tvalid[k])) return;
  const double d = c.d_src, zp = p.zpos;
  cd Pf[2], Pb[2];
  for (int m = 0; m < 2; ++m) {
    Pf[m] = cexp(mul_i(ldc(c.Qf, m, c.n, k)) * (d - zp));
    Pb[m] = cexp(mul_i(-ldc(c.Qb, m, c.n, k)) * zp);
  }
  cd T[4][4];
  for (int r = 0; r < 4; ++r)
    for (int cc = 0; cc < 4; ++cc) T[r][cc] = ldc(c.T, r + 4 * cc, c.n, k);
  for (int q = 0; q < 3; ++q) {
    cd sf0 = ldc(c.sf, 0 + 2 * q, c.n, k) * Pf[0], sf1 = ldc(c.sf, 1 + 2 * q, c.n, k) * Pf[1];
    cd sb0 = ldc(c.sb, 0 + 2 * q, c.n, k) * Pb[0], sb1 = ldc(c.sb, 1 + 2 * q, c.n, k) * Pb[1];
    // rows 0,1 (Af) use the F masks, rows 2,3 (Ab) the B masks
    cd uF[4] = {p.uf_F * sf0, p.uf_F * sf1, p.ub_F * sb0, p.ub_F * sb1};
    cd uB[4] = {p.uf_B * sf0, p.uf_B * sf1, p.ub_B * sb0, p.ub_B * sb1};
    for (int m = 0; m < 2; ++m) {
      cd a = T[m][0] * uF[0];
      a += T[m][1] * uF[1];
      a += T[m][2] * uF[2];
      a += T[m][3] * uF[3];
      Af[m][q] = a;
      cd b = T[2 + m][0] * uB[0];
      b += T[2 + m][1] * uB[1];
      b += T[2 + m][2] * uB[2];
      b += T[2 + m][3] * uB[3];
      Ab[m][q] = b;
    }
  }
}

// same-layer direct amplitudes at z_obs (direct_amplitude, :232-259), point source
__device__ __forceinline__ void direct_amp(const SynthParams& p, long k, double z, cd Afd[2][3], cd Abd[2][3]) {
  const CacheView& c = p.c;
  for (int m = 0; m < 2; ++m)
    for (int q = 0; q < 3; ++q) { Afd[m][q] = cd{0, 0}; Abd[m][q] = cd{0, 0}; }
  if (!c.valid[k]) return;
  const double zeta = z - p.zpos;
  if (zeta > 0) {
    for (int m = 0; m < 2; ++m) {
      cd e = phase_cl(ldc(c.Qf, m, c.n, k), zeta);
      for (int q = 0; q < 3; ++q) Afd[m][q] = ldc(c.sf, m + 2 * q, c.n, k) * e;
    }
  } else if (zeta < 0) {
    for (int m = 0; m < 2; ++m) {
      cd e = phase_cl(ldc(c.Qb, m, c.n, k), zeta);
      for (int q = 0; q < 3; ++q) Abd[m][q] = ldc(c.sb, m + 2 * q, c.n, k) * e;
    }
  }
}

// ------------------------------------------------------------------------------------
// 1D coefficients. Columns per z-row: order 0: xx yx xy yy zz; order 1: zx zy xz yz;
// order 2: xx yx xy yy (c q); stored: the 9 independent ones (store_coef_row, C1D_R* real rows
// per height). Output rows are real: row 2*(zi*ncol + col) + part, node fastest.
// ------------------------------------------------------------------------------------
// the 13 coefficient columns of one (node, z row) (_integrate_pixel_1d's integrand,
// mod_ClosedFormField.jl:435-487): order 0: xx yx xy yy zz; order 1: zx zy xz yz; order 2:
// xx yx xy yy
__device__ __forceinline__ void coef1d_row(const SynthParams& p, long k, double z, const cd Af[2][3], const cd Ab[2][3],
                                           cd c0[5], cd c1[4], cd c2[4]) {
  const CacheView& c = p.c;
  const long n = c.n;
  // i w / (2π) with a complex weight and node on a deformed contour (kri, wri), real otherwise
  const cd W = cd{0.0, 1.0 / (2.0 * 3.14159265358979323846)} * cd{c.wr[k], c.wri ? c.wri[k] : 0.0};
  const cd kx{c.kr[k], c.kri ? c.kri[k] : 0.0};
  for (int i = 0; i < 5; ++i) c0[i] = cd{0, 0};
  for (int i = 0; i < 4; ++i) { c1[i] = cd{0, 0}; c2[i] = cd{0, 0}; }
  cd Afd[2][3], Abd[2][3];
  if (p.with_direct) direct_amp(p, k, z, Afd, Abd);
  const cd half_i{0.0, 0.5};
  for (int m = 0; m < 2; ++m) {
    cd kzf = ldc(c.basis, 12 + m, n, k), kzb = ldc(c.basis, 14 + m, n, k);
    cd af[3], ab[3], gf, gb;
    if (p.with_direct) {
      cd pf = phase_cl(kzf, z), pb = phase_cl(kzb, z - p.d_obs);
      for (int q = 0; q < 3; ++q) {
        af[q] = fin0(W * (Afd[m][q] + Af[m][q] * pf));
        ab[q] = fin0(W * (Abd[m][q] + Ab[m][q] * pb));
      }
      gf = kx;
      gb = kx;
    } else {
      for (int q = 0; q < 3; ++q) { af[q] = fin0(W * Af[m][q]); ab[q] = fin0(W * Ab[m][q]); }
      gf = phase_cl(kzf, z) * kx;
      gb = phase_cl(kzb, z - p.d_obs) * kx;
    }
    for (int br = 0; br < 2; ++br) {
      const cd* a = br == 0 ? af : ab;
      cd g = br == 0 ? gf : gb;
      cd ex = ldc(c.basis, (br == 0 ? 0 : 6) + m, n, k);
      cd ey = ldc(c.basis, (br == 0 ? 2 : 8) + m, n, k);
      cd ez = ldc(c.basis, (br == 0 ? 4 : 10) + m, n, k);
      cd ax = a[0] * g, ay = a[1] * g, az = a[2] * g;
      // q = x: A = ax, B = ay
      c0[0] += half_i * (-(ax * ex) - ay * ey);  // xx
      c2[0] += half_i * (ax * ex - ay * ey);
      c0[1] += half_i * (-(ax * ey) + ay * ex);  // yx
      c2[1] += half_i * (ax * ey + ay * ex);
      c1[0] += ax * ez;                          // zx
      // q = y: A = ay, B = -ax
      c0[2] += half_i * (-(ay * ex) + ax * ey);  // xy
      c2[2] += half_i * (ay * ex + ax * ey);
      c0[3] += half_i * (-(ay * ey) - ax * ex);  // yy
      c2[3] += half_i * (ay * ey - ax * ex);
      c1[1] += ay * ez;                          // zy
      // q = z: C = az
      c1[2] += az * ex;                          // xz
      c1[3] += az * ey;                          // yz
      c0[4] += cd{0.0, -1.0} * (az * ez);        // zz
    }
  }
}

// the 9 stored complex columns of one (node, height) as real rows (C1D_R* per height) of
// C0, C1, C2 (row stride `stride`)
template <class T>
__device__ __forceinline__ void store_coef_row(T* C0, T* C1, T* C2, long stride, long k, int zi, const cd c0[5],
                                               const cd c1[4], const cd c2[4]) {
  const cd s0[3] = {c0[0], c0[1], c0[4]};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const long r = 2L * (zi * 3 + j);
    C0[r * stride + k] = (T)s0[j].x;
    C0[(r + 1) * stride + k] = (T)s0[j].y;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long r = 2L * (zi * 4 + j);
    C1[r * stride + k] = (T)c1[j].x;
    C1[(r + 1) * stride + k] = (T)c1[j].y;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const long r = 2L * (zi * 2 + j);
    C2[r * stride + k] = (T)c2[j].x;
    C2[(r + 1) * stride + k] = (T)c2[j].y;
  }
}

// the 13 order sums of one (radius, height) from the stored ones (Pn(col) = the complex value
// of stored column col of order n): yy = xx, xy = -yx of order 0; xy = yx, yy = -xx of order 2
template <class F0, class F1, class F2>
__device__ __forceinline__ void unpack_order_sums(F0 P0, F1 P1, F2 P2, cd g0[5], cd g1[4], cd g2[4]) {
  g0[0] = P0(0);
  g0[1] = P0(1);
  g0[2] = -g0[1];
  g0[3] = g0[0];
  g0[4] = P0(2);
#pragma unroll
  for (int j = 0; j < 4; ++j) g1[j] = P1(j);
  g2[0] = P2(0);
  g2[1] = P2(1);
  g2[2] = g2[1];
  g2[3] = -g2[0];
}

// J_0, J_1, J_2 of a real argument: power series below 1 (relative accuracy down to x = 0), the Taylor rows
// up to 25 (|error| <= 2e-16), Hankel's expansion with one phase for both orders above (the library past
// 1e15); J_2 from the recurrence (A&S 9.1.27) from 1 on.
// Bound by FP64 issue: 251 radii x 4081 nodes took 13.8 us with the library's j0 and j1, each with its own
// ranges and phase, and a J_2 series with twelve divisions; 9.9 us (error of the map 7e-15 -> 2e-15).
__device__ __forceinline__ void bessel_j012(double x, double& a0, double& a1, double& a2) {
  const double ax = fabs(x);
  if (ax < 1.0) {
    const double h2 = 0.25 * x * x;
    a0 = bessel_series_unit<0>(h2);
    a1 = 0.5 * x * bessel_series_unit<1>(h2);
    a2 = 0.5 * h2 * bessel_series_unit<2>(h2);
    return;
  }
  if (ax < (double)JTAB_N) {
    const int i = (int)ax;
    const double d = ax - ((double)i + 0.5);
    const double* c = JTAB + i * JTAB_M;
    double v = c[JTAB_M - 1], w = 0.0;
#pragma unroll
    for (int m = JTAB_M - 2; m >= 0; --m) {
      w = fma(w, d, v);
      v = fma(v, d, c[m]);
    }
    a0 = v;
    a1 = x < 0.0 ? w : -w;
  } else if (ax < 1e15) {
    const double y = 1.0 / ax, w = y * y;
    double sn, cs;
    sincos(ax, &sn, &cs);
    const double am = sqrt(y * 0.31830988618379067154);  // √(1 / (πx)): the phases' √½ taken in
    const double c0 = am * (cs + sn), s0 = am * (sn - cs);
    a0 = hankel_sum<0, 0>(w) * c0 - (y * hankel_sum<0, 1>(w)) * s0;
    a1 = hankel_sum<1, 0>(w) * s0 + (y * hankel_sum<1, 1>(w)) * c0;
    if (x < 0.0) a1 = -a1;
  } else {  // also Inf and NaN
    a0 = j0(x);
    a1 = j1(x);
  }
  a2 = (2.0 / x) * a1 - a0;
}

// Bessel tables J_n(k ρ), n = 0, 1, 2; row r = radius, k contiguous, rows ld apart
__global__ void k_bessel(const double* kr, long nk, const double* rho, int nr, long ld, double* J0, double* J1,
                         double* J2) {
  long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int r = blockIdx.y;
  if (k >= nk) return;
  double x = kr[k] * rho[r];
  long o = (long)r * ld + k;
  double a0, a1, a2;
  bessel_j012(x, a0, a1, a2);
  J0[o] = a0;
  J1[o] = a1;
  J2[o] = a2;
}

// largest of the warp's values max(|x|, |y|) as IEEE bits (non-negative doubles order as their bits),
// Inf where either is not finite: the high words first, then the low words of the lanes that hold the
// largest high one
__device__ __forceinline__ unsigned long long warp_max_bits(cd v, bool live) {
  unsigned hx = (unsigned)__double2hiint(v.x) & 0x7fffffffu, hy = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
  unsigned lx = (unsigned)__double2loint(v.x), ly = (unsigned)__double2loint(v.y);
  const bool y = hy > hx || (hy == hx && ly > lx);
  unsigned h = y ? hy : hx, l = y ? ly : lx;
  if (h >= 0x7ff00000u) { h = 0x7ff00000u; l = 0; }
  if (!live) h = l = 0;
  const unsigned mh = __reduce_max_sync(0xffffffffu, h);
  const unsigned ml = __reduce_max_sync(0xffffffffu, h == mh ? l : 0u);
  return (unsigned long long)mh << 32 | ml;
}

// J_n(kρ ρ) of complex nodes (deformed contour): real and imaginary tables of each order, rows ld apart.
// With rs (zeroed by the caller; [order][slice][radius] IEEE bits, slices of kchunk nodes, a multiple of
// 32) also each slice's largest |Re J| or |Im J|, reduced per warp.
__global__ void __launch_bounds__(128) k_bessel_c(const double* kr, const double* kri, long nk, const double* rho, int nr,
                                                  long ld, double* J, unsigned long long* rs, long kchunk, int nchunk) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  const bool live = k < nk;
  if (!live && !rs) return;
  cd a[3] = {cd{0.0, 0.0}, cd{0.0, 0.0}, cd{0.0, 0.0}};
  if (live) {
    const cd z = cd{kr[k], kri[k]} * rho[r];
    if (z.x == 0.0 && z.y == 0.0) a[0] = cd{1.0, 0.0};
    else bessel_j012_c(z, a[0], a[1], a[2]);
    const long o = (long)r * ld + k, plane = (long)nr * ld;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      J[2 * n * plane + o] = a[n].x;
      J[(2 * n + 1) * plane + o] = a[n].y;
    }
  }
  if (rs) {
    const int z = (int)(((long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) / kchunk);
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      // a NaN counts as no maximum
      const cd v{a[n].x == a[n].x ? a[n].x : 0.0, a[n].y == a[n].y ? a[n].y : 0.0};
      const unsigned long long bits = warp_max_bits(v, live);
      if ((threadIdx.x & 31) == 0 && z < nchunk) atomicMax(rs + ((long)n * nchunk + z) * nr + r, bits);
    }
  }
}

cudaError_t launch_bessel_c(const double* kr, const double* kri, long nk, const double* rho, int nr, long ld, double* J,
                            cudaStream_t s, unsigned long long* rs, long kchunk, int nchunk) {
  if (nk <= 0 || nr <= 0) return cudaSuccess;
  if (rs && (kchunk <= 0 || kchunk % 32 != 0)) return cudaErrorInvalidValue;
  dim3 grid((unsigned)((nk + 127) / 128), (unsigned)nr);
  k_bessel_c<<<grid, 128, 0, s>>>(kr, kri, nk, rho, nr, ld, J, rs, kchunk, nchunk);
  return cudaGetLastError();
}

// one complex J_n evaluation per thread (the device Bessel functions, exposed for testing)
__global__ void k_bessel_eval(long n, int order, const double* zr, const double* zi, double* outr, double* outi) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  cd a0, a1, a2;
  const cd z{zr[t], zi[t]};
  if (z.x == 0.0 && z.y == 0.0) {
    a0 = cd{1.0, 0.0}; a1 = cd{0.0, 0.0}; a2 = cd{0.0, 0.0};
  } else {
    bessel_j012_c(z, a0, a1, a2);
  }
  const cd v = order == 0 ? a0 : (order == 1 ? a1 : a2);
  outr[t] = v.x;
  outi[t] = v.y;
}

cudaError_t launch_bessel_eval(long n, int order, const double* zr, const double* zi, double* outr, double* outi,
                               cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_bessel_eval<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(n, order, zr, zi, outr, outi);
  return cudaGetLastError();
}

cudaError_t launch_bessel(const double* kr, long nk, const double* rho, int nr, long ld, double* J0, double* J1,
                          double* J2, cudaStream_t s) {
  dim3 grid((unsigned)((nk + 127) / 128), (unsigned)nr);
  k_bessel<<<grid, 128, 0, s>>>(kr, nk, rho, nr, ld, J0, J1, J2);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// FP64 contractions out[split][n][m] = Σ_k A[m][k] B[n][k] (both operands k-contiguous), up to six
// of them (the Bessel orders; real and imaginary J on a contour) in one grid, each cut into
// column tiles, row tiles and k slices; the pixel assembly sums the slices in order. FP64
// tensor-core instructions (mma m8n8k4: one operand load serves 8 rows or columns, where the
// scalar FMA tile it replaces was bound by its shared-memory loads and its load-compute-load
// barriers), a ring of 16-k stages filled by cp.async, warps of 32 x 32 or 16 x 16 outputs. Rows of
// a stage are 20 doubles apart, so the 4 x 4 operand words of a half-warp fall in distinct banks.
// Bound: the FP64 pipe (37 TFLOP/s) on large sets; the latency of the k chain on small ones, hence
// the 32 x 32 tile there, which gives more slices.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int G64_K = 16, G64_LD = 20, G64_STAGES = 3;

// BM x BN tile, WT x WT outputs per warp
template <int BM, int BN, int WT>
__global__ void __launch_bounds__(32 * (BM / WT) * (BN / WT)) k_gemm64(const __grid_constant__ Gemm64 p) {
  constexpr int WN = BN / WT, NT = 32 * (BM / WT) * WN, F = WT / 8;
  extern __shared__ __align__(16) double g64[];
  constexpr int STAGE = (BM + BN) * G64_LD;
  int e = 0;
  while (e + 1 < p.n && p.e[e + 1].first <= (int)blockIdx.x) ++e;
  const Gemm64Entry& E = p.e[e];
  const int ntm = (p.M + BM - 1) / BM, ntn = (E.N + BN - 1) / BN;
  const int u = (int)blockIdx.x - E.first;
  const int bm = (u % ntm) * BM, bn = (u / ntm % ntn) * BN, sp = u / (ntm * ntn);
  const long k0 = (long)sp * p.kchunk, k1 = min(p.K, k0 + p.kchunk);
  const int nst = k1 > k0 ? (int)((k1 - k0 + G64_K - 1) / G64_K) : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp / WN) * WT, wn = (warp % WN) * WT;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(g64);
  // one stage: (BM + BN) rows of 16 doubles, 8 copies of 16 bytes per row; rows past the operand
  // and k past the slice are zero-filled
  auto fill = [&](int st) {
    const long kk = k0 + (long)st * G64_K;
    const uint32_t base = sbase + (uint32_t)((st % G64_STAGES) * STAGE) * 8u;
    for (int t = tid; t < (BM + BN) * 8; t += NT) {
      const int row = t >> 3, c = 2 * (t & 7);
      const bool isa = row < BM;
      const int g = isa ? bm + row : bn + row - BM;
      const bool in = isa ? g < p.M : g < E.N;
      const long left = k1 - kk - c;
      const int bytes = in ? (left >= 2 ? 16 : left == 1 ? 8 : 0) : 0;
      const double* src = isa ? E.A + (bytes ? (long)g * p.lda + kk + c : 0) : E.B + (bytes ? (long)g * p.ldb + kk + c : 0);
      cp16(base + (uint32_t)(row * G64_LD + c) * 8u, src, bytes);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[F][F][2];
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int s = 0; s < G64_STAGES - 1; ++s) {
    if (s < nst) fill(s);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0; s < nst; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(G64_STAGES - 2) : "memory");
    __syncthreads();
    if (s + G64_STAGES - 1 < nst) fill(s + G64_STAGES - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const double* A = g64 + (s % G64_STAGES) * STAGE + (wm + (lane >> 2)) * G64_LD + (lane & 3);
    const double* B = g64 + (s % G64_STAGES) * STAGE + (BM + wn + (lane >> 2)) * G64_LD + (lane & 3);
#pragma unroll
    for (int q = 0; q < G64_K; q += 4) {
      double a[F], b[F];
#pragma unroll
      for (int i = 0; i < F; ++i) {
        a[i] = A[8 * i * G64_LD + q];
        b[i] = B[8 * i * G64_LD + q];
      }
#pragma unroll
      for (int i = 0; i < F; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j) mma_f64(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  double* out = E.out + (long)sp * E.N * p.M;
#pragma unroll
  for (int i = 0; i < F; ++i) {
    const int m = bm + wm + 8 * i + (lane >> 2);
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < F; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = bn + wn + 8 * j + 2 * (lane & 3) + h;
        if (n < E.N) out[(long)n * p.M + m] = acc[i][j][h];
      }
  }
}

// 128 x 64 tiles once they give 148 CTAs (251 radii x 61 heights x 4081 nodes: 55 us, 90 us with 32 x 32
// ones); below that 32 x 32 tiles, whose shorter warps and finer slices shorten the k chain (8 radii x 4
// heights x 256 nodes: 4.3 us against 9.3 us)
static bool gemm64_large(const Gemm64& p) {
  long t = 0;
  for (int i = 0; i < p.n; ++i) t += (long)((p.M + 127) / 128) * ((p.e[i].N + 63) / 64);
  return t * std::max(1L, p.K / 256) >= 148;
}

int gemm64_plan(Gemm64& p) {
  const bool big = gemm64_large(p);
  const int bm = big ? 128 : 32, bn = big ? 64 : 32;
  long tiles = 0;
  for (int i = 0; i < p.n; ++i) tiles += (long)((p.M + bm - 1) / bm) * ((p.e[i].N + bn - 1) / bn);
  // k slices that fill the SMs (two 128 x 64 or four 32 x 32 CTAs each), at least 64 nodes long
  const long want = std::max(1L, std::min((148L * (big ? 2 : 4)) / std::max(1L, tiles), p.K / 64));
  p.kchunk = ((p.K + want - 1) / want + G64_K - 1) / G64_K * G64_K;
  if (p.kchunk <= 0) p.kchunk = G64_K;
  p.splits = (int)std::max(1L, (p.K + p.kchunk - 1) / p.kchunk);
  return p.splits;
}

cudaError_t launch_gemm64(Gemm64 p, cudaStream_t s) {
  if (p.M <= 0 || p.n <= 0) return cudaSuccess;
  if ((p.lda | p.ldb) & 1) return cudaErrorInvalidValue;
  const bool big = gemm64_large(p);
  const int bm = big ? 128 : 32, bn = big ? 64 : 32;
  int blocks = 0;
  for (int i = 0; i < p.n; ++i) {
    p.e[i].first = blocks;
    blocks += ((p.M + bm - 1) / bm) * ((p.e[i].N + bn - 1) / bn) * p.splits;
  }
  const int smem = G64_STAGES * (bm + bn) * G64_LD * 8;
  if (big) {
    cudaError_t e = cudaFuncSetAttribute(k_gemm64<128, 64, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_gemm64<128, 64, 32><<<blocks, 256, smem, s>>>(p);
  } else {
    k_gemm64<32, 32, 16><<<blocks, 128, smem, s>>>(p);
  }
  return cudaGetLastError();
}

// acc[i] = (add ? acc[i] : 0) + Σ_z part[z][i], z in order
__global__ void k_sum_slices(long len, int nz, const double* __restrict__ part, double* __restrict__ acc, int add) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int z = 0; z < nz; ++z) s += part[(long)z * len + i];
    acc[i] = add ? acc[i] + s : s;
  }
}

cudaError_t launch_sum_slices(long len, int nz, const double* part, double* acc, int add, cudaStream_t s) {
  if (len <= 0) return cudaSuccess;
  k_sum_slices<<<(unsigned)std::min<long>((len + 255) / 256, 148L * 16), 256, 0, s>>>(len, nz, part, acc, add);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// 1D assembly: combine orders, rotate per pixel, Julia layout (Nx, Ny, Nz, 3, 3)
// obs-layer basis of one node: kz and the field components (E_f, E_b) of the two modes
__device__ __forceinline__ void load_obs_basis(const CacheView& c, long node, cd kzf[2], cd kzb[2], cd ef[2][3],
                                               cd eb[2][3]) {
  const long n = c.n;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    kzf[m] = ldc(c.basis, 12 + m, n, node);
    kzb[m] = ldc(c.basis, 14 + m, n, node);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ef[m][a] = ldc(c.basis, 2 * a + m, n, node);
      eb[m][a] = ldc(c.basis, 6 + 2 * a + m, n, node);
    }
  }
}

// the nine strengths of one (node, z row) (_strengths_row!, mod_ClosedFormField.jl:616-659):
// s[a][q] = Σ_m E_f[m][a] w (A_f[m][q] e^{i kzf z} + direct) + E_b[m][a] w (A_b ... )
__device__ __forceinline__ void strengths_row(const SynthParams& p, long node, double z, cd W, const cd Af[2][3],
                                              const cd Ab[2][3], const cd kzf[2], const cd kzb[2], const cd ef[2][3],
                                              const cd eb[2][3], cd s[3][3]) {
  // the direct term (direct_amp) is formed per mode inline: sf[m][q] e^{i Qf zeta} above the
  // source, sb[m][q] e^{i Qb zeta} below it, exact zeros elsewhere (as direct_amp's arrays)
  const CacheView& c = p.c;
  const double zeta = z - p.zpos;
  const bool dir = p.with_direct && c.valid[node];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) s[a][b] = cd{0, 0};
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const cd pf = phase_cl(kzf[m], z);
    const cd pb = phase_cl(kzb[m], z - p.d_obs);
    cd edf{0.0, 0.0}, edb{0.0, 0.0};
    const bool up = dir && zeta > 0, dn = dir && zeta < 0;
    if (up) edf = phase_cl(ldc(c.Qf, m, c.n, node), zeta);
    if (dn) edb = phase_cl(ldc(c.Qb, m, c.n, node), zeta);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      cd tf = Af[m][q] * pf, tb = Ab[m][q] * pb;
      if (p.with_direct) {
        tf += up ? ldc(c.sf, m + 2 * q, c.n, node) * edf : cd{0.0, 0.0};
        tb += dn ? ldc(c.sb, m + 2 * q, c.n, node) * edb : cd{0.0, 0.0};
      }
      const cd af = fin0(W * tf), ab = fin0(W * tb);
#pragma unroll
      for (int a = 0; a < 3; ++a) s[a][q] += ef[m][a] * af + eb[m][a] * ab;
    }
  }
}

// ------------------------------------------------------------------------------------
// one pixel of the 1D assembly: the order sums g0[5], g1[4], g2[4] of its radius combined
// into the 3x3 dyadic of the frame along the pixel's azimuth, then rotated to (x, y):
// G = Rot R Rotᵀ, written at pix + npix (zi + nz (cc + 3 q))
__device__ __forceinline__ void assemble1d_pixel(double x, double y, const cd g0[5], const cd g1[4], const cd g2[4],
                                                 long pix, long npix, int zi, int nz, double2* G) {
  cd R[3][3];
  R[0][0] = g0[0] + g2[0];
  R[1][0] = g0[1] + g2[1];
  R[2][0] = g1[0];
  R[0][1] = g0[2] + g2[2];
  R[1][1] = g0[3] + g2[3];
  R[2][1] = g1[1];
  R[0][2] = g1[2];
  R[1][2] = g1[3];
  R[2][2] = g0[4];
  double rho = hypot(x, y);
  double cp = rho == 0.0 ? 1.0 : x / rho, sp = rho == 0.0 ? 0.0 : y / rho;
  double Rot[3][3] = {{cp, -sp, 0.0}, {sp, cp, 0.0}, {0.0, 0.0, 1.0}};
  for (int q = 0; q < 3; ++q)
    for (int cc = 0; cc < 3; ++cc) {
      cd s{0, 0};
      for (int a = 0; a < 3; ++a) {
        cd tt = Rot[cc][0] * R[0][a] + Rot[cc][1] * R[1][a] + Rot[cc][2] * R[2][a];
        s += tt * Rot[q][a];
      }
      G[pix + npix * (zi + (long)nz * (cc + 3 * q))] = make_double2(s.x, s.y);
    }
}

// acc[j] = Σ_z p[z N M + j M], j < R, z = first, first + step, ...: the slices of one (radius, height)'s R
// real columns in order, all columns of a slice in flight together; with step 4 (ASM_SPLIT) the
// lanes 8 apart hold four interleaved parts of the slices, added at the end
template <int R>
__device__ __forceinline__ void sum_columns(const double* __restrict__ p, long M, long NM, int nchunk, int first, int step,
                                            double acc[R]) {
#pragma unroll
  for (int j = 0; j < R; ++j) acc[j] = 0.0;
  p += first * NM;
#pragma unroll 2
  for (int z = first; z < nchunk; z += step, p += step * NM)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[j] += __ldg(p + j * M);
  if (step > 1)
#pragma unroll
    for (int j = 0; j < R; ++j) {
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 8);
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
    }
}
// the order's complex columns of one (radius, height); on a deformed contour part holds Re J · C^T and
// part_im Im J · C^T of the real and imaginary columns
template <int R>
__device__ __forceinline__ void order_columns(const Asm1D& a, int o, int zi, int r, int first, int step, cd g[R / 2]) {
  const long M = a.nr, NM = (long)R * a.nz * M, off = (long)R * zi * M + r;
  double x[R];
  sum_columns<R>(a.part[o] + off, M, NM, a.nchunk, first, step, x);
#pragma unroll
  for (int c = 0; c < R / 2; ++c) g[c] = cd{x[2 * c], x[2 * c + 1]};
  if (a.part_im[o]) {
    sum_columns<R>(a.part_im[o] + off, M, NM, a.nchunk, first, step, x);
#pragma unroll
    for (int c = 0; c < R / 2; ++c) g[c] = cd{g[c].x - x[2 * c + 1], g[c].y + x[2 * c]};
  }
}

// one thread per (pixel, height), or four lanes of one warp (asm1d_split): the order sums of the pixel's
// radius, then the pixel assembly. Blocks of 128 threads; b: the block within the item.
__device__ __forceinline__ void assemble1d_body(const Asm1D& a, long b) {
  const long npix = (long)a.nx * a.ny;
  const int nz = a.nz, step = asm1d_split(a.nchunk);
  const int lane = threadIdx.x & 31;
  const int first = step > 1 ? lane >> 3 : 0;
  long t = step > 1 ? (b * 4 + (threadIdx.x >> 5)) * 8 + (lane & 7) : b * 128 + threadIdx.x;
  const bool live = t < npix * nz;
  if (!live) {
    if (step == 1) return;
    t = 0;  // the warp's shuffles need every lane
  }
  const long pix = t % npix;
  const int zi = (int)(t / npix);
  const int ix = (int)(pix % a.nx), iy = (int)(pix / a.nx);
  const int r = a.rmap[pix];
  cd g0[5], g1[4], g2[4];
  if (a.sym) {
    cd s0[C1S_R0 / 2], s1[C1S_R1 / 2], s2[C1S_R2 / 2];
    order_columns<C1S_R0>(a, 0, zi, r, first, step, s0);
    order_columns<C1S_R1>(a, 1, zi, r, first, step, s1);
    order_columns<C1S_R2>(a, 2, zi, r, first, step, s2);
    const cd z{0.0, 0.0};
    g0[0] = g0[3] = s0[0]; g0[1] = g0[2] = z; g0[4] = s0[1];
    g1[0] = s1[0]; g1[2] = s1[1]; g1[1] = g1[3] = z;
    g2[0] = s2[0]; g2[3] = -s2[0]; g2[1] = g2[2] = z;
  } else {
    cd s0[C1D_R0 / 2], s1[C1D_R1 / 2], s2[C1D_R2 / 2];
    order_columns<C1D_R0>(a, 0, zi, r, first, step, s0);
    order_columns<C1D_R1>(a, 1, zi, r, first, step, s1);
    order_columns<C1D_R2>(a, 2, zi, r, first, step, s2);
    unpack_order_sums([&](int c) { return s0[c]; }, [&](int c) { return s1[c]; }, [&](int c) { return s2[c]; }, g0, g1,
                      g2);
  }
  if (!live || first > 0) return;
  assemble1d_pixel(a.xs[ix], a.ys[iy], g0, g1, g2, pix, npix, zi, nz, a.G);
}

__global__ void __launch_bounds__(128) k_assemble1d(const __grid_constant__ Asm1D a) {
  assemble1d_body(a, blockIdx.x);
}

cudaError_t launch_assemble1d(const Asm1D& a, cudaStream_t s) {
  const long blocks = asm1d_blocks(a);
  if (blocks <= 0) return cudaSuccess;
  k_assemble1d<<<(unsigned)blocks, 128, 0, s>>>(a);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// 2D strengths per (node, z-row): S[col'][n], col' = zi + nz (c + 3q)
// One thread per (node, group of SG_Z z-rows): the reflected amplitudes (z-independent) and
// the mode basis are formed once per group. With `colmax` set, the kernel also reduces
// max(|Re S|, |Im S|) over each (node slice of `kchunk` nodes, column): a warp max (a warp's
// 32 nodes lie in one slice, kchunk being a multiple of 32) and one atomicMax per warp on
// the IEEE bits, which order like the values for non-negative doubles (Inf/NaN sort above
// every finite value, so a non-finite strength shows in the slice's maximum).
// ------------------------------------------------------------------------------------
constexpr int SG_Z = 8;  // z-rows per thread

__global__ void __launch_bounds__(128) k_strengths2d(SynthParams p, double2* S, unsigned long long* colmax, long kchunk) {
  const long nidx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const CacheView& c = p.c;
  const long n = c.n;
  const bool live = nidx < n;
  const long node = live ? nidx : n - 1;
  const long k = node % c.Nk, pp = node / c.Nk;
  const double w = c.kr[k] * c.wr[k] * c.wphi[pp] / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
  const cd W{w, 0.0};
  cd Af[2][3], Ab[2][3];
  reflected_amp(p, node, Af, Ab);
  cd kzf[2], kzb[2], ef[2][3], eb[2][3];
  load_obs_basis(c, node, kzf, kzb, ef, eb);
  const int z0 = blockIdx.y * SG_Z, z1 = min(p.nz, z0 + SG_Z);
  for (int zi = z0; zi < z1; ++zi) {
    cd s[3][3];
    strengths_row(p, node, p.zo[zi], W, Af, Ab, kzf, kzb, ef, eb, s);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        const long col = zi + (long)p.nz * (cc + 3 * q);
        if (live) S[col * n + nidx] = make_double2(s[cc][q].x, s[cc][q].y);
        if (colmax) {
          double m = live ? fmax(fabs(s[cc][q].x), fabs(s[cc][q].y)) : 0.0;
          if (live && !(isfinite(s[cc][q].x) && isfinite(s[cc][q].y))) m = __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
          // fmax drops a NaN operand; Inf (set above for any non-finite entry) survives
          if ((threadIdx.x & 31) == 0 && live)
            atomicMax(colmax + (nidx / kchunk) * (long)(9 * p.nz) + col, (unsigned long long)__double_as_longlong(m));
        }
      }
  }
}

// ------------------------------------------------------------------------------------
// The same strengths in two kernels, for callers that give a scratch array `amp`:
// k_reflect2d writes each node's reflected amplitudes (A_f, A_b: 12 complex, node fastest)
// once; k_strengths_rows stages 32 nodes' amplitudes, basis, seeds and q's in shared memory
// (coalesced, once per block), then each of its 4 warps takes every fourth z row of the 32
// nodes, one node per lane. The arithmetic per row is strengths_row's, in the same order.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 4) k_reflect2d(SynthParams p, double2* __restrict__ amp) {
  const long node = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long n = p.c.n;
  if (node >= n) return;
  cd Af[2][3], Ab[2][3];
  reflected_amp(p, node, Af, Ab);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      amp[(long)(3 * m + q) * n + node] = make_double2(Af[m][q].x, Af[m][q].y);
      amp[(long)(6 + 3 * m + q) * n + node] = make_double2(Ab[m][q].x, Ab[m][q].y);
    }
}

// 1D coefficient columns from the reflected amplitudes k_reflect2d wrote once per node (the
// amplitudes do not depend on the z row); the arithmetic per (node, row) is coef1d_row's
// heights per thread of k_coef1d_amp: a node's amplitudes are loaded once for COEF1D_ZB
// z rows (the per-row arithmetic and outputs are those of one row per thread)
constexpr int COEF1D_ZB = 4;

// T = double for the FP64 contraction; float for the int8x3 one, whose digit images need 24
// significant bits (an FP32 rounding of a column's value adds at most half a step of its
// fixed-point scale) and whose coefficient columns are then half the memory traffic
template <class T>
__global__ void __launch_bounds__(128) k_coef1d_amp(SynthParams p, const double2* __restrict__ amp, T* C0, T* C1,
                                                     T* C2, long cst) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long n = p.c.n;
  if (k >= n) return;
  cd Af[2][3], Ab[2][3];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      Af[m][q] = ldc(amp, 3 * m + q, n, k);
      Ab[m][q] = ldc(amp, 6 + 3 * m + q, n, k);
    }
  const int z0 = blockIdx.y * COEF1D_ZB;
  const int z1 = min(p.nz, z0 + COEF1D_ZB);
  for (int zi = z0; zi < z1; ++zi) {
    cd c0[5], c1[4], c2[4];
    coef1d_row(p, k, p.zo[zi], Af, Ab, c0, c1, c2);
    store_coef_row(C0, C1, C2, cst, k, zi, c0, c1, c2);
  }
}

// ------------------------------------------------------------------------------------
// The symmetric columns (c1d_rows). Factors per node, rows of n (W = i w / 2π, a = the amplitude of
// the moment, e = the mode field, k the node, f / b the forward and backward wave):
//   0, 1  T: -(i/2) W a_y e_y k of TE      2, 3  P: -(i/2) W a_x e_x k of TM
//   4, 5  W a_x e_z k of TM                6, 7  W a_z e_x k             8, 9  -i W a_z e_z k
//   10-13 kz of TE f, TE b, TM f, TM b     14-23 the direct term's T, P, ... (f above the source, b below)
// and per height, g the branch phases: xx of order 0 = Σ T g + Σ P g, of order 2 = Σ T g - Σ P g,
// zx = Σ (4, 5) g, xz = Σ (6, 7) g, zz = Σ (8, 9) g. About 60 FP64 operations per (node, height),
// against 350 for the nine general columns from the amplitudes, and 10 stored columns against 18:
// 325k nodes x 64 heights took 1083 us and take 278 us (bound by the 832 MB of columns written, 127 us
// at the copy rate, and the FP64 pipe).
// ------------------------------------------------------------------------------------
// A_y of the TE mode, A_x and A_z of the TM one, as reflected_amp's entries: one orientation after the other,
// the T rows of its mode alone. Bound by load latency: 65536 nodes 17.4 us with all twelve amplitudes (162
// registers), 12.0 us at four CTAs per SM; 32 film stacks, 325k nodes, 84 -> 79 us.
__device__ __forceinline__ void reflect_sym_body(const SynthParams& p, long k, double2* amp) {
  const CacheView& c = p.c;
  const long n = c.n;
  const cd W = cd{0.0, 1.0 / (2.0 * 3.14159265358979323846)} * cd{c.wr[k], c.wri ? c.wri[k] : 0.0};
  const cd kx{c.kr[k], c.kri ? c.kri[k] : 0.0};
  // which of the two modes is TE: the one with the larger E_y (the other's is zero)
  const bool te1 = norm2(ldc(c.basis, 3, n, k)) + norm2(ldc(c.basis, 9, n, k)) >
                   norm2(ldc(c.basis, 2, n, k)) + norm2(ldc(c.basis, 8, n, k));
  const int te = te1 ? 1 : 0, tm = 1 - te;
  cd A[2][3];
#pragma unroll
  for (int q = 0; q < 3; ++q) A[0][q] = A[1][q] = cd{0.0, 0.0};
  if (c.valid[k] && c.tvalid[k]) {
    cd P[4];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      P[m] = cexp(mul_i(ldc(c.Qf, m, n, k)) * (c.d_src - p.zpos));
      P[2 + m] = cexp(mul_i(-ldc(c.Qb, m, n, k)) * p.zpos);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int m = q == 1 ? te : tm;
      cd s[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = ldc(i < 2 ? c.sf : c.sb, (i & 1) + 2 * q, n, k) * P[i];
#pragma unroll
      for (int br = 0; br < 2; ++br)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          A[br][q] += ldc(c.T, 2 * br + m + 4 * i, n, k) * ((i < 2 ? (br ? p.uf_B : p.uf_F) : (br ? p.ub_B : p.ub_F)) * s[i]);
    }
  }
  auto put = [&](int row, cd v) { amp[(long)row * n + k] = make_double2(v.x, v.y); };
  const cd half{0.0, -0.5};
#pragma unroll
  for (int br = 0; br < 2; ++br) {
    const cd ey = ldc(c.basis, (br == 0 ? 2 : 8) + te, n, k);
    const cd ex = ldc(c.basis, (br == 0 ? 0 : 6) + tm, n, k), ez = ldc(c.basis, (br == 0 ? 4 : 10) + tm, n, k);
    auto factors = [&](int row, cd ax, cd ay, cd az) {
      // not finite: coef_sym_rows leaves the node to the general columns and their clamps
      const cd wx = W * ax * kx, wy = W * ay * kx, wz = W * az * kx;
      put(row + br, half * (wy * ey));
      put(row + 2 + br, half * (wx * ex));
      put(row + 4 + br, wx * ez);
      put(row + 6 + br, wz * ex);
      put(row + 8 + br, cd{0.0, -1.0} * (wz * ez));
    };
    factors(0, A[br][0], A[br][1], A[br][2]);
    if (p.with_direct) {
      const double2* sd = br == 0 ? c.sf : c.sb;
      const bool v = c.valid[k];
      const cd z{0.0, 0.0};
      factors(C1S_AMP, v ? ldc(sd, tm, n, k) : z, v ? ldc(sd, te + 2, n, k) : z, v ? ldc(sd, tm + 4, n, k) : z);
    }
    put(10 + br, ldc(c.basis, (br == 0 ? 12 : 14) + te, n, k));
    put(12 + br, ldc(c.basis, (br == 0 ? 12 : 14) + tm, n, k));
  }
}
__global__ void __launch_bounds__(128, 4) k_reflect_sym(SynthParams p, double2* __restrict__ amp) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < p.c.n) reflect_sym_body(p, k, amp);
}

template <class T>
__device__ __forceinline__ void store_sym_row(T* C0, T* C1, T* C2, long cst, long k, int zi, const cd c[5]) {
  const long r4 = 4L * zi, r2 = 2L * zi;
  C0[r4 * cst + k] = (T)c[0].x; C0[(r4 + 1) * cst + k] = (T)c[0].y;
  C0[(r4 + 2) * cst + k] = (T)c[1].x; C0[(r4 + 3) * cst + k] = (T)c[1].y;
  C1[r4 * cst + k] = (T)c[2].x; C1[(r4 + 1) * cst + k] = (T)c[2].y;
  C1[(r4 + 2) * cst + k] = (T)c[3].x; C1[(r4 + 3) * cst + k] = (T)c[3].y;
  C2[r2 * cst + k] = (T)c[4].x; C2[(r2 + 1) * cst + k] = (T)c[4].y;
}

// rows whose phases or factors leave the fast path's range: the general columns' arithmetic with its
// clamps, out of line
template <class T>
__device__ __noinline__ void coef_sym_exact(const SynthParams& p, long k, int z0, int z1, T* C0, T* C1, T* C2, long cst) {
  cd Af[2][3], Ab[2][3];
  reflected_amp(p, k, Af, Ab);
  for (int zi = z0; zi < z1; ++zi) {
    cd c0[5], c1[4], c2[4];
    coef1d_row(p, k, p.zo[zi], Af, Ab, c0, c1, c2);
    const cd c[5] = {c0[0], c0[4], c1[0], c1[2], c2[0]};
    store_sym_row(C0, C1, C2, cst, k, zi, c);
  }
}

// rows z0 .. z1 - 1 of one node. Evenly spaced heights (dz != 0): each branch phase by one complex
// product per row, e^{i kz (z + dz)} = e^{i kz z} e^{i kz dz}, where every exponent stays in
// [-600, 80] (no underflowed start, no overflow); other heights: one exponential per branch and row.
template <class T>
__device__ __forceinline__ void coef_sym_rows(const SynthParams& p, const double2* amp, long k, int z0, int z1, double dz,
                                              T* C0, T* C1, T* C2, long cst) {
  const long n = p.c.n;
  cd F[10], kz[4];  // kz: TE f, TE b, TM f, TM b
#pragma unroll
  for (int i = 0; i < 10; ++i) F[i] = ldc(amp, i, n, k);
#pragma unroll
  for (int i = 0; i < 4; ++i) kz[i] = ldc(amp, 10 + i, n, k);
  double zlo = p.zo[z0], zhi = zlo, big = fabs(zlo), lo = 0.0, hi = 0.0;
  for (int zi = z0 + 1; zi < z1; ++zi) {
    zlo = fmin(zlo, p.zo[zi]);
    zhi = fmax(zhi, p.zo[zi]);
    big += fabs(p.zo[zi]);  // the extremes pass over a NaN
  }
#pragma unroll
  for (int i = 0; i < 10; ++i) big += fabs(F[i].x) + fabs(F[i].y);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double s = i & 1 ? p.d_obs : 0.0;
    big += fabs(kz[i].x) * (fabs(zlo) + fabs(zhi) + fabs(s));  // not finite for a layer of infinite thickness
    const double a = -kz[i].y * (zlo - s), b = -kz[i].y * (zhi - s);
    lo = fmin(lo, fmin(a, b));
    hi = fmax(hi, fmax(a, b));
    if (p.with_direct) {  // ζ > 0 forward, ζ < 0 backward: the far end of the rows on that side
      const double zeta = i & 1 ? fmin(zlo - p.zpos, 0.0) : fmax(zhi - p.zpos, 0.0);
      lo = fmin(lo, -kz[i].y * zeta);
      hi = fmax(hi, -kz[i].y * zeta);
    }
    big += fabs(kz[i].y);
  }
  if (p.with_direct)
    for (int i = C1S_AMP; i < C1S_AMP_DIRECT; ++i) { const cd v = ldc(amp, i, n, k); big += fabs(v.x) + fabs(v.y); }
  if (!(big < 1e200 && hi <= 80.0)) {  // also any NaN
    coef_sym_exact(p, k, z0, z1, C0, C1, C2, cst);
    return;
  }
  const bool rec = dz != 0.0 && lo >= -600.0;
  cd step[4], g[4], gd[2];
  if (rec)
#pragma unroll
    for (int i = 0; i < 4; ++i) step[i] = phase_call(kz[i], dz);
  int side = 0;  // of the source: +1 above, -1 below, where gd holds the last row's direct phases
  for (int zi = z0; zi < z1; ++zi) {
    const double z = p.zo[zi];
    if (rec && zi > z0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = g[i] * step[i];
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = phase_call(kz[i], i & 1 ? z - p.d_obs : z);
    }
    cd t = F[0] * g[0], q = F[2] * g[2];
    cd c[5];
    t += F[1] * g[1];
    q += F[3] * g[3];
    c[2] = F[4] * g[2];
    c[2] += F[5] * g[3];
    c[3] = F[6] * g[2];
    c[3] += F[7] * g[3];
    c[1] = F[8] * g[2];
    c[1] += F[9] * g[3];
    if (p.with_direct) {
      const double zeta = z - p.zpos;
      const int now = zeta > 0 ? 1 : zeta < 0 ? -1 : 0, br = now < 0 ? 1 : 0;
      if (now != 0) {
        if (rec && now == side) {
          gd[0] = gd[0] * (br ? step[1] : step[0]);
          gd[1] = gd[1] * (br ? step[3] : step[2]);
        } else {
          gd[0] = phase_call(br ? kz[1] : kz[0], zeta);
          gd[1] = phase_call(br ? kz[3] : kz[2], zeta);
        }
        t += ldc(amp, C1S_AMP + br, n, k) * gd[0];
        q += ldc(amp, C1S_AMP + 2 + br, n, k) * gd[1];
        c[2] += ldc(amp, C1S_AMP + 4 + br, n, k) * gd[1];
        c[3] += ldc(amp, C1S_AMP + 6 + br, n, k) * gd[1];
        c[1] += ldc(amp, C1S_AMP + 8 + br, n, k) * gd[1];
      }
      side = now;
    }
    c[0] = t + q;
    c[4] = t - q;
    store_sym_row(C0, C1, C2, cst, k, zi, c);
  }
}

// Three CTAs per SM: 65536 nodes x 256 rows 244 us at four (156 bytes of spills a thread), 210 us at three;
// 4081 x 61 in FP64 12.3 -> 9.1 us
template <class T>
__global__ void __launch_bounds__(128, 3) k_coef_sym(SynthParams p, const double2* __restrict__ amp, T* C0, T* C1, T* C2,
                                                     long cst, double dz, int zb) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= p.c.n) return;
  const int z0 = blockIdx.y * zb;
  coef_sym_rows(p, amp, k, z0, min(p.nz, z0 + zb), dz, C0, C1, C2, cst);
}

// the order-0 rows at C, orders 1 and 2 behind them
template <class T>
static cudaError_t coef1d_amp_impl(const SynthParams& p, double2* amp, T* C, long ldc, double dz, cudaStream_t s) {
  if (p.c.n <= 0 || p.nz <= 0) return cudaSuccess;
  if (p.sym) {
    const unsigned nb = (unsigned)((p.c.n + 127) / 128);
    T* C1 = C + (size_t)C1S_R0 * p.nz * ldc;
    k_reflect_sym<<<nb, 128, 0, s>>>(p, amp);
    // rows per thread: fewer where the grid fills less than a quarter of the SMs, whose time is the chain of
    // one thread's rows (256 nodes x 4 rows: 6.8 us at 16 rows a thread, 5.4 us at one); beyond that the
    // exponentials a split repeats cost more (4081 x 61: 9.1 us at 16 rows, 12.8 us at 8)
    int zb = COEF_SYM_ZB;
    while (zb > 1 && (long)nb * ((p.nz + zb - 1) / zb) < 37) zb /= 2;
    k_coef_sym<T><<<dim3(nb, (unsigned)((p.nz + zb - 1) / zb)), 128, 0, s>>>(
        p, amp, C, C1, C1 + (size_t)C1S_R1 * p.nz * ldc, ldc, dz, zb);
    return cudaGetLastError();
  }
  k_reflect2d<<<(unsigned)((p.c.n + 127) / 128), 128, 0, s>>>(p, amp);
  k_coef1d_amp<T><<<dim3((unsigned)((p.c.n + 127) / 128), (unsigned)((p.nz + COEF1D_ZB - 1) / COEF1D_ZB)), 128, 0, s>>>(
      p, amp, C, C + (size_t)C1D_OFF1 * p.nz * ldc, C + (size_t)C1D_OFF2 * p.nz * ldc, ldc);
  return cudaGetLastError();
}

cudaError_t launch_coef1d_amp(const SynthParams& p, double2* amp, double* C, long ldc, double dz, cudaStream_t s) {
  return coef1d_amp_impl<double>(p, amp, C, ldc, dz, s);
}

cudaError_t launch_coef1d_amp(const SynthParams& p, double2* amp, float* C, long ldc, double dz, cudaStream_t s) {
  return coef1d_amp_impl<float>(p, amp, C, ldc, dz, s);
}

// z rows zo[0 .. m - 1] evenly spaced (to 4 ulp of the progression); every lane of the warp calls it
__device__ __forceinline__ bool even_rows(const double* zo, int m, int lane, double& dz) {
  const double z0 = zo[0], z1 = zo[m - 1];
  dz = m > 1 ? (z1 - z0) / (m - 1) : 0.0;
  const double tol = 4 * 2.220446049250313e-16 * fmax(fabs(z0), fabs(z1));
  bool ok = m > 1 && isfinite(dz) && dz != 0.0;
  for (int r = lane; r < m; r += 32) ok = ok && fabs(zo[r] - (z0 + r * dz)) <= tol;
  return __all_sync(0xffffffffu, ok);
}

// per node of a k_strengths_rows block: 12 amplitudes, the obs-layer basis (16), sf, sb (6 each),
// Qf, Qb (2 each)
constexpr int SR_F = 44;
// phases per node: 0-3 the group's first row of mode 0 f, b, mode 1 f, b; 4-7 one row's step; 8-9 the
// direct term's first row above the source of modes 0, 1, 10-11 below it; 12-15 four rows' step
constexpr int SR_P = 16, SR_ROWS = 32;
// One block per 32 nodes, each of its 4 warps every fourth z row, one node per lane. Evenly spaced rows
// take their phases by complex products, e^{i kz (z + dz)} = e^{i kz z} e^{i kz dz}, from exponentials
// that the warps share out per group of 32 rows (12 per node; one per phase and row before, six per
// row with the direct term), where every exponent of the group stays in [-600, 80]; other rows and
// nodes take phase_cl. 65536 nodes x 8 rows with the direct term: 51 us against 87 us with an exponential per
// phase and row, synchronous staging, shuffled FP64 maxima and a division per column.
// At most 128 registers: four CTAs per SM.
__global__ void __launch_bounds__(128, 4) k_strengths_rows(SynthParams p, const double2* __restrict__ amp,
                                                         double2* __restrict__ S, unsigned long long* colmax,
                                                         long kchunk) {
  __shared__ double2 sh[SR_F][32];
  __shared__ double2 ph[SR_P][32];
  const CacheView& c = p.c;
  const long n = c.n;
  const long node0 = (long)blockIdx.x * 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // stage the 32 nodes' inputs: field f of node node0 + j at sh[f][j] (coalesced over j; asynchronous
  // copies, so that the eleven loads of a thread are in flight together)
  for (int e = tid; e < SR_F * 32; e += 128) {
    const int j = e & 31, f = e >> 5;
    const long node = min(node0 + j, n - 1);
    const double2* src = f < 12 ? amp + f * n : f < 28 ? c.basis + (f - 12) * n : f < 34 ? c.sf + (f - 28) * n
                       : f < 40 ? c.sb + (f - 34) * n : f < 42 ? c.Qf + (f - 40) * n : c.Qb + (f - 42) * n;
    cp16((uint32_t)__cvta_generic_to_shared(&sh[f][j]), reinterpret_cast<const double*>(src + node), 16);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // every warp forms the nodes' weights; 32-bit division where the node count allows
  const long nd = min(node0 + lane, n - 1);
  const long pp = n <= 0x7fffffffL ? (long)((unsigned)nd / (unsigned)c.Nk) : nd / c.Nk, k = nd - pp * c.Nk;
  const double W = c.kr[k] * c.wr[k] * c.wphi[pp] / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
  const bool dir = p.with_direct && c.valid[nd];
  unsigned long long* cmax = colmax ? colmax + (node0 / kchunk) * (long)(9 * p.nz) : nullptr;
  double dz;
  const bool even = even_rows(p.zo, p.nz, lane, dz);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the weight into the amplitudes and the direct term's seeds (fields 0-11 and 28-39)
  for (int f = warp; f < 24; f += 4) {
    double2& v = sh[f < 12 ? f : f + 16][lane];
    v = make_double2(W * v.x, W * v.y);
  }
  __syncthreads();
  const long nidx = node0 + lane;
  const bool live = nidx < n;
  auto g = [&](int f) { const double2 v = sh[f][lane]; return cd{v.x, v.y}; };
  auto gp = [&](int f) { const double2 v = ph[f][lane]; return cd{v.x, v.y}; };
  auto kz = [&](int i) { return g(i & 1 ? 26 + (i >> 1) : 24 + (i >> 1)); };  // mode i >> 1, f (0) or b (1)
  bool stepped = false;  // this node's steps are in ph (written by the first group that takes the recurrence)
  for (int zg = 0; zg < p.nz; zg += SR_ROWS) {
    const int ng = min(SR_ROWS, p.nz - zg);
    bool rec = false;
    int u0 = 0, d0 = 0;  // the group's first rows above and below the source
    if (even) {
      const double zr = p.zo[zg + min(lane, ng - 1)], z0 = p.zo[zg], z1 = p.zo[zg + ng - 1];
      const unsigned up = __ballot_sync(0xffffffffu, lane < ng && zr > p.zpos);
      const unsigned dn = __ballot_sync(0xffffffffu, lane < ng && zr < p.zpos);
      u0 = up ? __ffs(up) - 1 : 0;
      d0 = dn ? __ffs(dn) - 1 : 0;
      double lo = 0.0, hi = 0.0, big = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const cd k = kz(i);
        const double s = i & 1 ? p.d_obs : 0.0;
        const double a = -k.y * (z0 - s), b = -k.y * (z1 - s);
        lo = fmin(lo, fmin(a, b));
        hi = fmax(hi, fmax(a, b));
        if (p.with_direct) {  // the far end of the rows on the wave's side
          const double far = i & 1 ? fmin(fmin(z0, z1) - p.zpos, 0.0) : fmax(fmax(z0, z1) - p.zpos, 0.0);
          lo = fmin(lo, -k.y * far);
          hi = fmax(hi, -k.y * far);
        }
        big += fabs(k.x) * (fabs(z0) + fabs(z1) + fabs(s)) + fabs(k.y);
      }
      rec = lo >= -600.0 && hi <= 80.0 && big < 1e200;  // false for any NaN
      if (rec) {
        const double zu = p.zo[zg + u0] - p.zpos, zd = p.zo[zg + d0] - p.zpos;
#pragma unroll 1
        for (int e = warp; e < 12; e += 4) {
          const int i = e < 8 ? e & 3 : e < 10 ? 2 * (e - 8) : 2 * (e - 10) + 1;
          const double at = e < 4 ? (i & 1 ? z0 - p.d_obs : z0) : e < 8 ? dz : e < 10 ? zu : zd;
          if ((e >= 4 && e < 8 && stepped) || (e >= 8 && !p.with_direct)) continue;
          const cd v = phase_call(kz(i), at);
          ph[e][lane] = make_double2(v.x, v.y);
          if (e >= 4 && e < 8) {
            cd q = v * v;
            q = q * q;
            ph[8 + e][lane] = make_double2(q.x, q.y);
          }
        }
        stepped = true;
      }
    }
    __syncthreads();
    cd gr[4], gd[2];
    if (rec)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        gr[i] = gp(i);
        for (int r = 0; r < warp; ++r) gr[i] = gr[i] * gp(4 + i);
      }
    int side = 0;
    for (int r = warp; r < ng; r += 4) {
      const int zi = zg + r;
      const double z = p.zo[zi];
      const double zeta = z - p.zpos;
      const bool up = dir && zeta > 0, dn = dir && zeta < 0;
      if (rec) {
        if (r > warp)
#pragma unroll
          for (int i = 0; i < 4; ++i) gr[i] = gr[i] * gp(12 + i);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) gr[i] = phase_cl(kz(i), i & 1 ? z - p.d_obs : z);
      }
      const int now = up ? 1 : dn ? -1 : 0, br = dn ? 1 : 0;
      if (now != 0) {
        if (!rec) {
          gd[0] = phase_cl(g(40 + 2 * br), zeta);
          gd[1] = phase_cl(g(41 + 2 * br), zeta);
        } else if (now == side) {
          gd[0] = gd[0] * gp(12 + br);
          gd[1] = gd[1] * gp(14 + br);
        } else {
          gd[0] = gp(8 + 2 * br);
          gd[1] = gp(9 + 2 * br);
          for (int q = br ? d0 : u0; q < r; ++q) {
            gd[0] = gd[0] * gp(4 + br);
            gd[1] = gd[1] * gp(6 + br);
          }
        }
      }
      side = now;
      cd s[3][3];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) s[a][b] = cd{0, 0};
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const cd pf = gr[2 * m], pb = gr[2 * m + 1];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          cd tf = g(3 * m + q) * pf, tb = g(6 + 3 * m + q) * pb;
          if (up) tf += g(28 + m + 2 * q) * gd[m];
          if (dn) tb += g(34 + m + 2 * q) * gd[m];
          const cd af = fin0(tf), ab = fin0(tb);
#pragma unroll
          for (int a = 0; a < 3; ++a) s[a][q] += g(12 + 2 * a + m) * af + g(18 + 2 * a + m) * ab;
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          const int col = zi + p.nz * (cc + 3 * q);
          if (live) S[col * n + nidx] = make_double2(s[cc][q].x, s[cc][q].y);
          if (cmax) {
            const unsigned long long bits = warp_max_bits(s[cc][q], live);
            if (lane == 0) atomicMax(cmax + col, bits);
          }
        }
    }
    __syncthreads();
  }
}

cudaError_t launch_strengths2d(const SynthParams& p, double2* S, cudaStream_t s, unsigned long long* colmax, long kchunk,
                               double2* amp) {
  if (p.c.n <= 0) return cudaSuccess;
  if (colmax && (kchunk <= 0 || kchunk % 32 != 0)) return cudaErrorInvalidValue;
  if (amp) {
    k_reflect2d<<<(unsigned)((p.c.n + 127) / 128), 128, 0, s>>>(p, amp);
    k_strengths_rows<<<(unsigned)((p.c.n + 31) / 32), 128, 0, s>>>(p, amp, S, colmax, kchunk);
    return cudaGetLastError();
  }
  dim3 grid((unsigned)((p.c.n + 127) / 128), (unsigned)((p.nz + SG_Z - 1) / SG_Z));
  k_strengths2d<<<grid, 128, 0, s>>>(p, S, colmax, kchunk);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// 2D lateral sum: G[pix][col] = Σ_n e^{i(kx_n x_i + ky_n y_j)} S[col][n] (complex FP64), for callers
// without room for phase tables (ytf_green_noalloc)
// Tile: 64 pixels x 32 columns, 16 nodes per stage; 256 threads, 4 pixels x 2 columns each.
// The phase operand is generated per stage in shared memory (sincos per node and
// coordinate, then one complex product per (node, pixel)).
// ------------------------------------------------------------------------------------
constexpr int LP = 64, LC = 32, LK = 16;
__global__ void __launch_bounds__(256) k_lateral(CacheView c, int nx, int ny, const double* __restrict__ xs,
                                                 const double* __restrict__ ys, int ncol, const double2* __restrict__ S,
                                                 double2* __restrict__ Gp, long kchunk) {
  __shared__ double2 Ps[LK][LP];
  __shared__ double2 Ss[LK][LC];
  __shared__ double kxs[LK], kys[LK];
  const long npix = (long)nx * ny;
  const long p0 = (long)blockIdx.x * LP;
  const int c0 = blockIdx.y * LC;
  const int sp = blockIdx.z;
  const long n = c.n;
  const long k0 = (long)sp * kchunk, k1 = min(n, k0 + kchunk);
  const int tid = threadIdx.x;
  const int tp = tid % 16, tc = tid / 16;  // pixels tp + 16 a (a < 4), columns tc + 16 b (b < 2)
  double2 acc[4][2];
  for (int a = 0; a < 4; ++a)
    for (int b = 0; b < 2; ++b) acc[a][b] = make_double2(0.0, 0.0);
  for (long kk = k0; kk < k1; kk += LK) {
    if (tid < LK) {
      long nn = kk + tid;
      double kx = 0.0, ky = 0.0;
      if (nn < k1) {
        long k = nn % c.Nk, q = nn / c.Nk;
        double s, co;
        sincos(c.phi[q], &s, &co);
        kx = c.kr[k] * co;
        ky = c.kr[k] * s;
      }
      kxs[tid] = kx;
      kys[tid] = ky;
    }
    __syncthreads();
    // phases: LK x LP = 1024 products, 4 per thread
    for (int e = 0; e < 4; ++e) {
      int idx = tid + 256 * e;
      int t = idx / LP, pl = idx % LP;
      long pix = p0 + pl;
      double2 v = make_double2(0.0, 0.0);
      if (pix < npix && kk + t < k1) {
        int i = (int)(pix % nx), j = (int)(pix / nx);
        double sx, cx, sy, cy;
        sincos(kxs[t] * xs[i], &sx, &cx);
        sincos(kys[t] * ys[j], &sy, &cy);
        v = make_double2(cx * cy - sx * sy, cx * sy + sx * cy);
      }
      Ps[t][pl] = v;
    }
    // strengths: LK x LC = 512, 2 per thread
    for (int e = 0; e < 2; ++e) {
      int idx = tid + 256 * e;
      int t = idx % LK, cl = idx / LK;
      long nn = kk + t;
      int col = c0 + cl;
      Ss[t][cl] = (nn < k1 && col < ncol) ? S[(long)col * n + nn] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < LK; ++t) {
      double2 pv[4], sv[2];
      for (int a = 0; a < 4; ++a) pv[a] = Ps[t][tp + 16 * a];
      for (int b = 0; b < 2; ++b) sv[b] = Ss[t][tc + 16 * b];
      for (int a = 0; a < 4; ++a)
        for (int b = 0; b < 2; ++b) {
          acc[a][b].x = fma(pv[a].x, sv[b].x, fma(-pv[a].y, sv[b].y, acc[a][b].x));
          acc[a][b].y = fma(pv[a].x, sv[b].y, fma(pv[a].y, sv[b].x, acc[a][b].y));
        }
    }
    __syncthreads();
  }
  double2* G = Gp + (long)sp * npix * ncol;
  for (int a = 0; a < 4; ++a) {
    long pix = p0 + tp + 16 * a;
    if (pix >= npix) continue;
    for (int b = 0; b < 2; ++b) {
      int col = c0 + tc + 16 * b;
      if (col < ncol) G[pix + npix * col] = acc[a][b];
    }
  }
}

// ------------------------------------------------------------------------------------
// The same sum on the FP64 tensor-core instructions, for callers with room for the phase tables
// Ex[i][n] = e^{i kx_n x_i}, Ey[j][n] = e^{i ky_n y_j} (k_phase_tables64, one sincos per node and
// coordinate): real form G[pix][2c + part] = Σ_k A[pix][k] B[k][2c + part] over k = 2 n + {0, 1}, A =
// (Re P, Im P) with P = Ex Ey formed once per stage of 8 nodes, B = (Sr, -Si) for the real and (Si, Sr)
// for the imaginary column, read from the strengths themselves with the sign flipped on load. A CTA
// of four warps takes 64 pixels x 8 F real columns (F <= 12: all 4 F columns of most calls, so P is
// formed once per pixel), one node slice; a warp 16 pixels x all columns.
//   Bound: the FP64 pipe. 576 pixels x 36 columns x 49152 nodes: 307 us (26.6 TFLOP/s); k_lateral, which
// takes two sincos per (node, pixel, 32 columns) and 6 shared loads per 8 products, 1189 us.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_phase_tables64(CacheView c, int nx, int ny, const double* __restrict__ xs,
                                                        const double* __restrict__ ys, double2* __restrict__ Ex,
                                                        double2* __restrict__ Ey, long n0, long n) {
  const long nn = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (nn >= n) return;
  double sp, cp;
  sincos(c.phi[(n0 + nn) / c.Nk], &sp, &cp);
  const double k = c.kr[(n0 + nn) % c.Nk];
  // rows of each axis split over blockIdx.y
  for (int e = blockIdx.y; e < nx + ny; e += gridDim.y) {
    double s, co;
    sincos(e < nx ? k * cp * xs[e] : k * sp * ys[e - nx], &s, &co);
    (e < nx ? Ex + (long)e * n : Ey + (long)(e - nx) * n)[nn] = make_double2(co, s);
  }
}

constexpr int L64_P = 64, L64_N = 8, L64_LD = 2 * L64_N + 4;

template <int F>
__global__ void __launch_bounds__(128, F <= 9 ? 3 : 2) k_lateral64(const __grid_constant__ Lateral64 p) {
  constexpr int NC = 4 * F;  // complex columns
  __shared__ __align__(16) double As[2][L64_P * L64_LD];
  __shared__ __align__(16) double Bs[2][NC * L64_LD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long p0 = (long)blockIdx.x * L64_P;
  const int c0 = blockIdx.y * NC;
  const long k0 = (long)blockIdx.z * p.kchunk, k1 = min(p.n, k0 + p.kchunk);
  const int nst = (int)((k1 - k0 + L64_N - 1) / L64_N);
  // the phase products of this thread: node tid & 7 of pixels (tid >> 3) + 16 e
  const double2 *ex[4], *ey[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const long pix = min(p0 + (tid >> 3) + 16 * e, p.npix - 1);  // a pixel past the set repeats the last
    ex[e] = p.Ex + (pix % p.nx) * p.n;
    ey[e] = p.Ey + (pix / p.nx) * p.n;
  }
  double2 px[4], py[4];
  auto load_phases = [&](int st) {
    const long nn = min(k0 + (long)st * L64_N + (tid & 7), p.n - 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      px[e] = __ldg(ex[e] + nn);
      py[e] = __ldg(ey[e] + nn);
    }
  };
  auto store_phases = [&](int st) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      *reinterpret_cast<double2*>(&As[st & 1][((tid >> 3) + 16 * e) * L64_LD + 2 * (tid & 7)]) =
          make_double2(px[e].x * py[e].x - px[e].y * py[e].y, px[e].x * py[e].y + px[e].y * py[e].x);
  };
  // strengths of 8 nodes per column, zero past the slice and the columns (so that what A holds there
  // does not count)
  auto load_strengths = [&](int st) {
    for (int t = tid; t < NC * L64_N; t += 128) {
      const int c = t >> 3, j = t & 7;
      const long nn = k0 + (long)st * L64_N + j;
      const bool in = c0 + c < p.ncol && nn < k1;
      cp16((uint32_t)__cvta_generic_to_shared(&Bs[st & 1][c * L64_LD + 2 * j]),
           reinterpret_cast<const double*>(p.S + (in ? (long)(c0 + c) * p.lds + nn : 0)), in ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[2][F][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  // B fragment of a lane: column (lane >> 2) of 8 real ones = complex column >> 1, part & 1; k = lane & 3
  const int part = (lane >> 2) & 1, kp = lane & 1;
  const int flip = (part == 0 && kp == 1) ? (int)0x80000000 : 0;
  const int boff = (lane >> 3) * L64_LD + 2 * ((lane & 3) >> 1) + (part ^ kp);
  const int aoff = (16 * warp + (lane >> 2)) * L64_LD + (lane & 3);
  if (nst > 0) {
    load_phases(0);
    load_strengths(0);
    store_phases(0);
  }
  for (int st = 0; st < nst; ++st) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (st + 1 < nst) {
      load_phases(st + 1);
      load_strengths(st + 1);
    }
    const double* A = As[st & 1] + aoff;
    const double* B = Bs[st & 1] + boff;
#pragma unroll
    for (int q = 0; q < 2 * L64_N; q += 4) {
      const double a0 = A[q], a1 = A[8 * L64_LD + q];
#pragma unroll
      for (int j = 0; j < F; ++j) {
        const double v = B[4 * j * L64_LD + q];
        const double b = __hiloint2double(__double2hiint(v) ^ flip, __double2loint(v));
        mma_f64(acc[0][j][0], acc[0][j][1], a0, b);
        mma_f64(acc[1][j][0], acc[1][j][1], a1, b);
      }
    }
    if (st + 1 < nst) store_phases(st + 1);
  }
  double2* G = p.partial + (long)blockIdx.z * p.npix * p.ncol;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const long pix = p0 + 16 * warp + 8 * i + (lane >> 2);
    if (pix >= p.npix) continue;
#pragma unroll
    for (int j = 0; j < F; ++j) {
      const int c = c0 + 4 * j + (lane & 3);
      if (c < p.ncol) G[pix + p.npix * c] = make_double2(acc[i][j][0], acc[i][j][1]);
    }
  }
}

// nodes per pass: phase tables of at most 1 GiB, or of one 8-node stage where the coordinates are that many
long lateral64_pass(long n, int nx, int ny) {
  const long fit = (1L << 30) / (16L * ((long)nx + ny)) / L64_N * L64_N;
  return std::min(n, std::max(fit, (long)L64_N));
}

// balanced column tiles of at most 48 complex columns
static int lateral64_f(int ncol) {
  const int tiles = (ncol + 47) / 48;
  return ((ncol + tiles - 1) / tiles + 3) / 4;
}

int lateral64_plan(Lateral64& p) {
  const int nc = 4 * lateral64_f(p.ncol);
  const long tiles = ((p.npix + L64_P - 1) / L64_P) * ((p.ncol + nc - 1) / nc);
  // node slices for three CTAs per SM, at least 64 nodes each
  const long want = std::max(1L, std::min(148L * 3 / tiles, p.n / 64));
  p.kchunk = ((p.n + want - 1) / want + L64_N - 1) / L64_N * L64_N;
  p.splits = (int)((p.n + p.kchunk - 1) / p.kchunk);
  return p.splits;
}

template <int F>
static void lateral64_run(const Lateral64& p, cudaStream_t s) {
  if constexpr (F >= 1) {
    if (lateral64_f(p.ncol) != F) return lateral64_run<F - 1>(p, s);
    const dim3 grid((unsigned)((p.npix + L64_P - 1) / L64_P), (unsigned)((p.ncol + 4 * F - 1) / (4 * F)),
                    (unsigned)p.splits);
    k_lateral64<F><<<grid, 128, 0, s>>>(p);
  }
}

cudaError_t launch_lateral64(const Lateral64& p, const CacheView& c, const double* xs, const double* ys, cudaStream_t s) {
  if (p.npix <= 0 || p.ncol <= 0 || p.n <= 0) return cudaSuccess;
  const int ny = (int)(p.npix / p.nx);
  k_phase_tables64<<<dim3((unsigned)((p.n + 127) / 128), (unsigned)std::min(p.nx + ny, 8)), 128, 0, s>>>(
      c, p.nx, ny, xs, ys, p.Ex, p.Ey, p.n0, p.n);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  lateral64_run<12>(p, s);
  return cudaGetLastError();
}

// Σ_k P[k len] in the order of k, eight values in flight together
__device__ __forceinline__ double2 sum_in_order(const double2* __restrict__ P, long len, int n) {
  double2 s = make_double2(0.0, 0.0);
  for (int k = 0; k < n; k += 8) {
    double2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k + i < n) v[i] = __ldg(P + (long)(k + i) * len);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k + i < n) {
        s.x += v[i].x;
        s.y += v[i].y;
      }
  }
  return s;
}
// One thread per output; bound by the chain of its loads: 12285 outputs 14.6 us with one load at a
// time in blocks of 256, 7.6 us; 20736 outputs 8.0 -> 5.1 us
__global__ void __launch_bounds__(64) k_reduce_splits2(long len, int splits, const double2* __restrict__ P,
                                                       double2* __restrict__ C, int add) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  double2 s = sum_in_order(P + i, len, splits);
  if (add) {
    const double2 c = C[i];
    s = make_double2(c.x + s.x, c.y + s.y);
  }
  C[i] = s;
}

int lateral_splits(long n, int splits) {
  long kchunk = (n + splits - 1) / splits;
  kchunk = ((kchunk + LK - 1) / LK) * LK;
  if (kchunk <= 0) return 1;
  return (int)std::max(1L, (n + kchunk - 1) / kchunk);
}

cudaError_t launch_lateral(const CacheView& c, int nx, int ny, const double* xs, const double* ys, int ncol, const double2* S,
                           double2* partial, int splits, cudaStream_t s) {
  long npix = (long)nx * ny;
  splits = lateral_splits(c.n, splits);
  long kchunk = (c.n + splits - 1) / splits;
  kchunk = ((kchunk + LK - 1) / LK) * LK;
  dim3 grid((unsigned)((npix + LP - 1) / LP), (unsigned)((ncol + LC - 1) / LC), (unsigned)splits);
  k_lateral<<<grid, 256, 0, s>>>(c, nx, ny, xs, ys, ncol, S, partial, kchunk);
  return cudaGetLastError();
}

cudaError_t launch_reduce_splits2(long len, int splits, const double2* partial, double2* G, cudaStream_t s, int add) {
  if (len <= 0) return cudaSuccess;
  k_reduce_splits2<<<(unsigned)((len + 63) / 64), 64, 0, s>>>(len, splits, partial, G, add);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// gl_rule panel expansion (mod_KxGrid.jl:361-384), no FMA contraction: bit-exact with a
// CPU evaluation of the same expressions in IEEE double
// ------------------------------------------------------------------------------------
__global__ void k_gl_nodes(int npanels, const double* pa, const double* pb, const int* sing_side, const double* xi,
                           const double* wx, int order, double* nodes, double* wts) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)npanels * order) return;
  int pi = (int)(t / order), j = (int)(t % order);
  double a = pa[pi], b = pb[pi];
  int sg = sing_side[pi];  // 0 regular, +1 singular at a, -1 singular at b
  if (sg == 0) {
    double h = __dmul_rn(0.5, __dsub_rn(b, a));
    double cc = __dmul_rn(0.5, __dadd_rn(a, b));
    nodes[t] = __dadd_rn(cc, __dmul_rn(h, xi[j]));
    wts[t] = __dmul_rn(h, wx[j]);
  } else {
    double L = sg > 0 ? a : b;
    double U = __dsqrt_rn(__dsub_rn(b, a));
    double hU = __dmul_rn(0.5, U);
    double u = __dmul_rn(hU, __dadd_rn(1.0, xi[j]));
    nodes[t] = __dadd_rn(L, __dmul_rn((double)sg, __dmul_rn(u, u)));
    wts[t] = __dmul_rn(__dmul_rn(hU, wx[j]), __dmul_rn(2.0, u));
  }
}

cudaError_t launch_gl_nodes(int npanels, const double* pa, const double* pb, const int* sing_side, const double* xi,
                            const double* wx, int order, double* nodes, double* wts, cudaStream_t s) {
  long tot = (long)npanels * order;
  if (tot == 0) return cudaSuccess;
  k_gl_nodes<<<(unsigned)((tot + 127) / 128), 128, 0, s>>>(npanels, pa, pb, sing_side, xi, wx, order, nodes, wts);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Batched synthesis of many small observation sets (uneven batches, one graph launch).
// Work unit = (item, chunk of nodes), pulled by persistent CTAs from a counter. Per sub-batch of
// SYN_SB = 32 nodes (one per lane) the CTA's four warps form in shared memory
//   first the phases of every z row (mode, forward / backward, direct) and of the source, rows and
//   exponentials dealt out over the warps;
//   then 2D: the strengths S[node][col] (col = zi + nz (cc + 3 q)), one source orientation q per warp,
//   and the pixels' phases e^{i kx x} e^{i ky y} (one sincos per x and per y) on the fourth;
//   or 1D: the real coefficient columns C[col][node], one group of columns per warp where TE and TM
//   decouple (5 complex columns per row: c1s), every fourth row per warp otherwise (13 per row), and
//   the tables J_n(kρ ρ_r), n = 0, 1, 2;
// then the outputs o = row + nrow col of the item's partial sum (2D rows: pixels, complex columns; 1D
// rows: distinct radii, real columns) take the sub-batch in register tiles of 4 rows x 3 (2D) or 1 (1D)
// columns, small sets with the nodes split over 2 or 4 groups of warps. k_synth_finish sums the chunks
// of each output in chunk order (2D) or sums them and assembles the pixel (1D).
// Bound by FP64 latency and issue. 96 uneven items, 266k nodes, 16 pixels x 4 rows each: 487 us with 64 nodes
// on two of the four warps (one thread through all of a node's strengths), 13 columns and one output
// per thread, two CTAs per SM; 245 us (349 with two CTAs per SM and no prefetch).
// ------------------------------------------------------------------------------------
constexpr int SYN_SB = 32, SYN_LD = SYN_SB + 1;

// the shared arrays of one item's work unit (bytes from the start), laid out with the item's own sizes
struct SynLayout {
  int nrow, ncol, units, groups;  // outputs, register tiles, node groups
  int acc, cols, tab, ph, bytes;
};
__host__ __device__ __forceinline__ SynLayout syn_layout(int is2d, int sym, int npix, int nr, int nz) {
  SynLayout L;
  L.nrow = is2d ? npix : nr;
  L.ncol = is2d ? 9 * nz : (sym ? 10 : 26) * nz;
  L.units = (L.nrow + 3) / 4 * (is2d ? (L.ncol + 2) / 3 : L.ncol);
  L.groups = L.units <= 32 ? 4 : L.units <= 64 ? 2 : 1;
  L.acc = 0;
  L.cols = L.groups * L.nrow * L.ncol * (is2d ? 16 : 8);
  L.cols = (L.cols + 15) / 16 * 16;
  L.tab = L.cols + (is2d ? SYN_SB * (L.ncol | 1) * 16 : L.ncol * SYN_LD * 8);
  L.tab = (L.tab + 15) / 16 * 16;
  L.ph = L.tab + (is2d ? SYN_SB * (npix | 1) * 16 : 3 * nr * SYN_LD * 8);
  L.ph = (L.ph + 15) / 16 * 16;
  L.bytes = L.ph + (6 * nz + 4) * SYN_SB * 16;
  return L;
}

size_t synth_small_smem(int is2d, int sym, int npix, int nr, int nz) {
  return (size_t)syn_layout(is2d, sym, npix, nr, nz).bytes;
}

size_t synth_small_smem() {
  const size_t a = synth_small_smem(1, 0, SYN_MAXPIX, 0, SYN_MAXZ), b = synth_small_smem(0, 0, 0, SYN_MAXR, SYN_MAXZ);
  return a > b ? a : b;
}

__device__ __forceinline__ int find_item(const long* __restrict__ off, int nb, long t) {
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// reflected amplitudes of source orientation q (reflected_amp, the source phases P: f 0, f 1, b 0, b 1)
__device__ __forceinline__ void reflected_amp_q(const SynthParams& p, long k, int q, const cd P[4], cd Af[2], cd Ab[2]) {
  const CacheView& c = p.c;
  Af[0] = Af[1] = Ab[0] = Ab[1] = cd{0.0, 0.0};
  if (!(c.valid[k] && c.tvalid[k])) return;
  const cd sf0 = ldc(c.sf, 2 * q, c.n, k) * P[0], sf1 = ldc(c.sf, 1 + 2 * q, c.n, k) * P[1];
  const cd sb0 = ldc(c.sb, 2 * q, c.n, k) * P[2], sb1 = ldc(c.sb, 1 + 2 * q, c.n, k) * P[3];
  const cd uF[4] = {p.uf_F * sf0, p.uf_F * sf1, p.ub_F * sb0, p.ub_F * sb1};
  const cd uB[4] = {p.uf_B * sf0, p.uf_B * sf1, p.ub_B * sb0, p.ub_B * sb1};
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Af[m] += ldc(c.T, m + 4 * i, c.n, k) * uF[i];
      Ab[m] += ldc(c.T, 2 + m + 4 * i, c.n, k) * uB[i];
    }
}

// phases of one sub-batch, [row][lane]: 6 zi + 2 m + (0 forward, 1 backward) of mode m, 6 zi + 4 + m the
// direct term's (forward above the source, backward below); 6 nz + i the source's P[i]
__device__ __forceinline__ void syn_phases(const SynthParams& p, long node, int warp, int lane, double2* ph) {
  const CacheView& c = p.c;
  const long n = c.n;
  for (int zi = warp; zi < p.nz; zi += 4) {
    const double z = p.zo[zi], zeta = z - p.zpos;
#pragma unroll 1
    for (int e = 0; e < 6; ++e) {
      if (e >= 4 && (!p.with_direct || zeta == 0.0)) continue;
      const int m = e >= 4 ? e - 4 : e >> 1;
      const bool b = e >= 4 ? zeta < 0.0 : (e & 1) != 0;
      const cd kz = e >= 4 ? ldc(b ? c.Qb : c.Qf, m, n, node) : ldc(c.basis, (b ? 14 : 12) + m, n, node);
      const double d = e >= 4 ? zeta : b ? z - p.d_obs : z;
      const cd v = phase_cl(kz, d);
      ph[(6 * zi + e) * SYN_SB + lane] = make_double2(v.x, v.y);
    }
  }
  const int m = warp & 1;
  const cd q = warp < 2 ? mul_i(ldc(c.Qf, m, n, node)) * (c.d_src - p.zpos) : mul_i(-ldc(c.Qb, m, n, node)) * p.zpos;
  const cd v = cexp(q);
  ph[(6 * p.nz + warp) * SYN_SB + lane] = make_double2(v.x, v.y);
}

// the next sub-batch's node data into L2 (48 rows, four 128-byte lines each of 32 nodes)
__device__ __forceinline__ void syn_prefetch(const CacheView& c, long node0, int tid) {
  for (int e = tid; e < 48 * 4; e += 128) {
    const int f = e >> 2;
    const long node = min(node0 + 8 * (e & 3), c.n - 1);
    const double2* src = f < 16 ? c.T + f * c.n : f < 32 ? c.basis + (f - 16) * c.n : f < 38 ? c.sf + (f - 32) * c.n
                       : f < 44 ? c.sb + (f - 38) * c.n : f < 46 ? c.Qf + (f - 44) * c.n : c.Qb + (f - 46) * c.n;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(src + node));
  }
}

// one orientation q of strengths_row at every z row of the node
__device__ __forceinline__ void syn_strengths(const SynthParams& p, long node, int lane, int q, const double2* ph, cd* S) {
  const CacheView& c = p.c;
  const long n = c.n;
  auto gp = [&](int f) { const double2 v = ph[f * SYN_SB + lane]; return cd{v.x, v.y}; };
  const int nz = p.nz;
  cd Af[2], Ab[2];
  {
    const cd P[4] = {gp(6 * nz), gp(6 * nz + 1), gp(6 * nz + 2), gp(6 * nz + 3)};
    reflected_amp_q(p, node, q, P, Af, Ab);
  }
  const long pp = n <= 0x7fffffffL ? (long)((unsigned)node / (unsigned)c.Nk) : node / c.Nk, k = node - pp * c.Nk;
  const double W = c.kr[k] * c.wr[k] * c.wphi[pp] / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
  const bool dir = p.with_direct && c.valid[node];
  cd ef[2][3], eb[2][3], sf[2], sb[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ef[m][a] = ldc(c.basis, 2 * a + m, n, node);
      eb[m][a] = ldc(c.basis, 6 + 2 * a + m, n, node);
    }
    sf[m] = sb[m] = cd{0.0, 0.0};
    if (dir) {
      sf[m] = ldc(c.sf, m + 2 * q, n, node);
      sb[m] = ldc(c.sb, m + 2 * q, n, node);
    }
  }
  for (int zi = 0; zi < nz; ++zi) {
    const double zeta = p.zo[zi] - p.zpos;
    cd s[3] = {cd{0.0, 0.0}, cd{0.0, 0.0}, cd{0.0, 0.0}};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      cd tf = Af[m] * gp(6 * zi + 2 * m), tb = Ab[m] * gp(6 * zi + 2 * m + 1);
      if (dir && zeta > 0.0) tf += sf[m] * gp(6 * zi + 4 + m);
      if (dir && zeta < 0.0) tb += sb[m] * gp(6 * zi + 4 + m);
      const cd af = fin0(cd{W, 0.0} * tf), ab = fin0(cd{W, 0.0} * tb);
#pragma unroll
      for (int a = 0; a < 3; ++a) s[a] += ef[m][a] * af + eb[m][a] * ab;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) S[zi + nz * (a + 3 * q)] = s[a];
  }
}

// decoupled TE / TM: the columns of one warp at every z row (coef1d_row's xx of orders 0 and 2 on warp 0,
// zx, xz, zz on warps 1, 2, 3), real and imaginary parts in rows of C
__device__ __forceinline__ void syn_columns_sym(const SynthParams& p, long node, int warp, int lane, const double2* ph,
                                                double* C) {
  const CacheView& c = p.c;
  const long n = c.n;
  auto gp = [&](int f) { const double2 v = ph[f * SYN_SB + lane]; return cd{v.x, v.y}; };
  const int nz = p.nz;
  const cd W = cd{0.0, 1.0 / (2.0 * 3.14159265358979323846)} * cd{c.wr[node], c.wri ? c.wri[node] : 0.0};
  const cd kx{c.kr[node], c.kri ? c.kri[node] : 0.0};
  // which of the two modes is TE: the one with the larger E_y (the other's is zero)
  const bool te1 = norm2(ldc(c.basis, 3, n, node)) + norm2(ldc(c.basis, 9, n, node)) >
                   norm2(ldc(c.basis, 2, n, node)) + norm2(ldc(c.basis, 8, n, node));
  const bool dir = p.with_direct && c.valid[node];
  const cd P[4] = {gp(6 * nz), gp(6 * nz + 1), gp(6 * nz + 2), gp(6 * nz + 3)};
  const cd half{0.0, -0.5};
  // term t: 0 TE of y, 1 TM of x or z; amplitudes, field factors kx e and direct seeds
  cd A[2][2], e[2][2], sd[2][2];
  int md[2];
  const int nt = warp == 0 ? 2 : 1;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (t >= nt) break;
    const bool teterm = warp == 0 && t == 0;
    const int q = teterm ? 1 : warp < 2 ? 0 : 2;
    md[t] = teterm == te1 ? 1 : 0;
    cd Af[2], Ab[2];
    reflected_amp_q(p, node, q, P, Af, Ab);
    A[t][0] = md[t] ? Af[1] : Af[0];
    A[t][1] = md[t] ? Ab[1] : Ab[0];
    const int comp = teterm ? 2 : warp == 0 || warp == 2 ? 0 : 4;  // E_y, E_x or E_z of the mode
    const cd f = warp == 0 ? half * kx : warp == 3 ? cd{0.0, -1.0} * kx : kx;
#pragma unroll
    for (int br = 0; br < 2; ++br) {
      e[t][br] = f * ldc(c.basis, 6 * br + comp + md[t], n, node);
      sd[t][br] = dir ? ldc(br ? c.sb : c.sf, md[t] + 2 * q, n, node) : cd{0.0, 0.0};
    }
  }
  for (int zi = 0; zi < nz; ++zi) {
    const double zeta = p.zo[zi] - p.zpos;
    cd v[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (t >= nt) break;
      const cd gf = gp(6 * zi + 2 * md[t]), gb = gp(6 * zi + 2 * md[t] + 1);
      if (p.with_direct) {
        cd tf = A[t][0] * gf, tb = A[t][1] * gb;
        if (dir && zeta > 0.0) tf += sd[t][0] * gp(6 * zi + 4 + md[t]);
        if (dir && zeta < 0.0) tb += sd[t][1] * gp(6 * zi + 4 + md[t]);
        v[t] = fin0(W * tf) * e[t][0] + fin0(W * tb) * e[t][1];
      } else {
        v[t] = (fin0(W * A[t][0]) * gf) * e[t][0] + (fin0(W * A[t][1]) * gb) * e[t][1];
      }
    }
    auto put = [&](int m, cd x) {
      C[(10 * zi + 2 * m) * SYN_LD + lane] = x.x;
      C[(10 * zi + 2 * m + 1) * SYN_LD + lane] = x.y;
    };
    if (warp == 0) {
      put(0, v[0] + v[1]);
      put(4, v[0] - v[1]);
    } else {
      put(warp == 1 ? 2 : warp == 2 ? 3 : 1, v[0]);
    }
  }
}

// acc (rows x cols of tile u; tw columns per tile) += the nodes t0 .. t1 - 1
template <int TW, class Row, class Col, class T>
__device__ __forceinline__ void syn_tile(int u, int nrow, int ncol, int t0, int t1, const Row& row, const Col& col, T* acc) {
  const int nrt = (nrow + 3) / 4;
  const int nct = (ncol + TW - 1) / TW;
  // real columns run over the lanes, complex tiles keep a column's row tiles together
  const int rt = TW == 1 ? u / nct : u % nrt, ct = TW == 1 ? u % nct : u / nrt;
  const int r0 = 4 * rt, c0 = TW * ct;
  T a[4][TW];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TW; ++j) a[i][j] = acc[min(r0 + i, nrow - 1) + nrow * min(c0 + j, ncol - 1)];
  for (int t = t0; t < t1; ++t) {
    T x[4], y[TW];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = row(t, min(r0 + i, nrow - 1), c0);
#pragma unroll
    for (int j = 0; j < TW; ++j) y[j] = col(t, min(c0 + j, ncol - 1));
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < TW; ++j) {
        if constexpr (TW == 1) {
          a[i][j] = fma(x[i], y[j], a[i][j]);
        } else {
          a[i][j].x = fma(x[i].x, y[j].x, fma(-x[i].y, y[j].y, a[i][j].x));
          a[i][j].y = fma(x[i].x, y[j].y, fma(x[i].y, y[j].x, a[i][j].y));
        }
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TW; ++j)
      if (r0 + i < nrow && c0 + j < ncol) acc[r0 + i + nrow * (c0 + j)] = a[i][j];
}

__global__ void __launch_bounds__(128, 3) k_synth_small(const SynthItem* __restrict__ items, int nitems,
                                                      const long* __restrict__ w_off, long nwork, unsigned* counter,
                                                      int chunk) {
  extern __shared__ __align__(16) unsigned char syn_smem[];
  __shared__ long wsh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (;;) {
    if (tid == 0) wsh = (long)atomicAdd(counter, 1u);
    __syncthreads();
    const long w = wsh;
    __syncthreads();
    if (w >= nwork) return;
    const int it = find_item(w_off, nitems, w);
    const SynthItem& I = items[it];
    const SynthParams& p = I.sp;
    const CacheView& c = p.c;
    const long cid = w - w_off[it];
    const long k0 = cid * chunk, k1 = min(c.n, k0 + chunk);
    const int nz = p.nz, npix = I.nx * I.ny;
    const bool two = I.is2d != 0;
    const SynLayout L = syn_layout(two, p.sym, npix, I.nr, nz);
    const int nout = L.nrow * L.ncol, nreal = two ? 2 * nout : nout;
    double* acc = reinterpret_cast<double*>(syn_smem + L.acc);     // [groups][ncol][nrow], 2D complex
    cd* Ss = reinterpret_cast<cd*>(syn_smem + L.cols);             // 2D [SB][ncol | 1]
    cd* Ps = reinterpret_cast<cd*>(syn_smem + L.tab);              // 2D [SB][npix | 1]
    double* Cs = reinterpret_cast<double*>(syn_smem + L.cols);     // 1D [ncol][SB + 1]
    double* Js = reinterpret_cast<double*>(syn_smem + L.tab);      // 1D [3][nr][SB + 1]
    double2* ph = reinterpret_cast<double2*>(syn_smem + L.ph);     // [6 nz + 4][SB]
    for (int o = tid; o < L.groups * nreal; o += 128) acc[o] = 0.0;
    for (long b0 = k0; b0 < k1; b0 += SYN_SB) {
      const int nb = (int)min((long)SYN_SB, k1 - b0);
      const long node = min(b0 + lane, k1 - 1);  // lanes past the end repeat the last node, and are not summed
      if (b0 + SYN_SB < k1) syn_prefetch(c, b0 + SYN_SB, tid);
      syn_phases(p, node, warp, lane, ph);
      __syncthreads();  // the phases are in, the last sub-batch is summed
      if (two) {
        if (warp < 3) {
          syn_strengths(p, node, lane, warp, ph, Ss + lane * (L.ncol | 1));
        } else {
          const long pp = c.n <= 0x7fffffffL ? (long)((unsigned)node / (unsigned)c.Nk) : node / c.Nk, k = node - pp * c.Nk;
          double sn, cs;
          sincos(c.phi[pp], &sn, &cs);
          const double kx = c.kr[k] * cs, ky = c.kr[k] * sn;
          cd* P = Ps + lane * (npix | 1);
          for (int jj = 0; jj < I.ny; ++jj) {  // e^{i ky y} in the row's last pixel, read before it is written
            double s2, c2;
            sincos(ky * I.ys[jj], &s2, &c2);
            P[I.nx * jj + I.nx - 1] = cd{c2, s2};
          }
          for (int i = 0; i < I.nx; ++i) {
            double sx, cx;
            sincos(kx * I.xs[i], &sx, &cx);
            for (int jj = 0; jj < I.ny; ++jj) {
              const cd y = P[I.nx * jj + I.nx - 1];
              P[i + I.nx * jj] = cd{cx * y.x - sx * y.y, cx * y.y + sx * y.x};
            }
          }
        }
      } else {
        if (p.sym) {
          syn_columns_sym(p, node, warp, lane, ph, Cs);
        } else if (warp < nz) {
          cd Af[2][3], Ab[2][3];
          reflected_amp(p, node, Af, Ab);
          for (int zi = warp; zi < nz; zi += 4) {
            cd cc[13];
            coef1d_row(p, node, p.zo[zi], Af, Ab, cc, cc + 5, cc + 9);
#pragma unroll
            for (int m = 0; m < 13; ++m) {
              Cs[(26 * zi + 2 * m) * SYN_LD + lane] = cc[m].x;
              Cs[(26 * zi + 2 * m + 1) * SYN_LD + lane] = cc[m].y;
            }
          }
        }
        const double kx = c.kr[node];
        for (int r = 3 - warp; r < I.nr; r += 4) {  // warp 0 has the most columns: it comes last
          double a0, a1, a2;
          bessel_j012(kx * I.rho[r], a0, a1, a2);
          Js[r * SYN_LD + lane] = a0;
          Js[(I.nr + r) * SYN_LD + lane] = a1;
          Js[(2 * I.nr + r) * SYN_LD + lane] = a2;
        }
      }
      __syncthreads();
      // groups of nodes: 4 of 32 threads, 2 of 64 or all 128 threads on all nodes
      const int gt = 128 / L.groups, g = tid / gt, per = SYN_SB / L.groups;
      const int t0 = g * per, t1 = min(nb, t0 + per);
      for (int u = tid - g * gt; u < L.units; u += gt) {
        if (two) {
          const int pld = npix | 1, sld = L.ncol | 1;
          syn_tile<3>(u, L.nrow, L.ncol, t0, t1, [&](int t, int r, int) { return Ps[t * pld + r]; },
                      [&](int t, int cidx) { return Ss[t * sld + cidx]; }, reinterpret_cast<cd*>(acc) + g * nout);
        } else {
          const int R = p.sym ? 10 : 26, h1 = p.sym ? 4 : 10, h2 = p.sym ? 8 : 18, nr = I.nr;
          syn_tile<1>(u, L.nrow, L.ncol, t0, t1,
                      [&](int t, int r, int cidx) {
                        const int h = cidx % R;
                        return Js[((h < h1 ? 0 : h < h2 ? nr : 2 * nr) + r) * SYN_LD + t];
                      },
                      [&](int t, int cidx) { return Cs[cidx * SYN_LD + t]; }, acc + g * nout);
        }
      }
    }
    __syncthreads();
    double* out = reinterpret_cast<double*>(I.partial) + cid * (long)nreal;
    for (int o = tid; o < nreal; o += 128) {
      double v = acc[o];
      for (int g = 1; g < L.groups; ++g) v += acc[g * nreal + o];
      out[o] = v;
    }
    __syncthreads();
  }
}

// x[m] = Σ_k part[k R nz nr + m nr], the chunks in order, four (R = 10) or two of them in flight together
template <int R>
__device__ __forceinline__ void sum_columns_in_order(const double* __restrict__ part, int nr, int nz, int nw, double x[R]) {
  constexpr int U = R > 16 ? 2 : 4;
  const long nout = (long)nr * R * nz;
#pragma unroll
  for (int m = 0; m < R; ++m) x[m] = 0.0;
  for (int k = 0; k < nw; k += U) {
    double v[U][R];
#pragma unroll
    for (int i = 0; i < U; ++i)
#pragma unroll
      for (int m = 0; m < R; ++m) v[i][m] = k + i < nw ? __ldg(part + (k + i) * nout + (long)m * nr) : 0.0;
#pragma unroll
    for (int i = 0; i < U; ++i)
#pragma unroll
      for (int m = 0; m < R; ++m) x[m] += v[i][m];
  }
}

// One thread per output (2D) or pixel (1D); bound by the chain of its loads over the chunks: 96 items 30 us
// with one chunk at a time, 10 us
__global__ void __launch_bounds__(64) k_synth_finish(const SynthItem* __restrict__ items, int nitems,
                                                       const long* __restrict__ f_off, long nfin) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nfin) return;
  const int it = find_item(f_off, nitems, t);
  const SynthItem& I = items[it];
  const long u = t - f_off[it];
  const int nz = I.sp.nz;
  const long npix = (long)I.nx * I.ny;
  if (I.is2d) {
    const long nout = npix * 9 * nz;
    I.G[u] = sum_in_order(I.partial + u, nout, I.nw);
    return;
  }
  const long pix = u % npix;
  const int zi = (int)(u / npix);
  const int r = I.rmap[pix];
  const int R = I.sp.sym ? 10 : 26;
  const double* part = reinterpret_cast<const double*>(I.partial) + r + (long)I.nr * R * zi;
  cd g[13];
  if (I.sp.sym) {
    double x[10];
    sum_columns_in_order<10>(part, I.nr, nz, I.nw, x);
    const cd z{0.0, 0.0}, c0{x[0], x[1]}, c4{x[8], x[9]};
    g[0] = g[3] = c0; g[1] = g[2] = z; g[4] = cd{x[2], x[3]};
    g[5] = cd{x[4], x[5]}; g[7] = cd{x[6], x[7]}; g[6] = g[8] = z;
    g[9] = c4; g[12] = -c4; g[10] = g[11] = z;
  } else {
    double x[26];
    sum_columns_in_order<26>(part, I.nr, nz, I.nw, x);
#pragma unroll
    for (int m = 0; m < 13; ++m) g[m] = cd{x[2 * m], x[2 * m + 1]};
  }
  const int i = (int)(pix % I.nx), j = (int)(pix / I.nx);
  assemble1d_pixel(I.xs[i], I.ys[j], g, g + 5, g + 9, pix, npix, zi, nz, I.G);
}

cudaError_t synth_small_init() {
  return cudaFuncSetAttribute(k_synth_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)synth_small_smem());
}

cudaError_t launch_synth_small(const SynthItem* items, int nitems, const long* w_off, long nwork, unsigned* counter,
                               int chunk, int grid, size_t smem, cudaStream_t s) {
  if (nwork <= 0) return cudaSuccess;
  if (grid <= 0 || chunk <= 0 || smem > synth_small_smem()) return cudaErrorInvalidValue;
  k_synth_small<<<grid, 128, smem, s>>>(items, nitems, w_off, nwork, counter, chunk);
  return cudaGetLastError();
}

cudaError_t launch_synth_finish(const SynthItem* items, int nitems, const long* f_off, long nfin, cudaStream_t s) {
  if (nfin <= 0) return cudaSuccess;
  k_synth_finish<<<(unsigned)((nfin + 63) / 64), 64, 0, s>>>(items, nitems, f_off, nfin);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Grouped 1D synthesis (int8x3 path): the reflected amplitudes, the FP32 coefficient columns
// and the final slice sum + pixel assembly of every item of a group, one launch each. The
// per-node and per-pixel arithmetic is that of k_reflect2d, k_coef1d_amp and k_assemble1d.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 4) k_reflect2d_group(const Synth1DItem* __restrict__ items,
                                                            const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const Synth1DItem& it = items[i];
  const long n = it.sp.c.n;
  const long node = (long)(blockIdx.x - first[i]) * blockDim.x + threadIdx.x;
  if (node >= n) return;
  cd Af[2][3], Ab[2][3];
  reflected_amp(it.sp, node, Af, Ab);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      it.amp[(long)(3 * m + q) * n + node] = make_double2(Af[m][q].x, Af[m][q].y);
      it.amp[(long)(6 + 3 * m + q) * n + node] = make_double2(Ab[m][q].x, Ab[m][q].y);
    }
}

// a read-only load the compiler keeps in place (volatile asm: not hoisted out of the row loop),
// so the node's mode fields are re-read from L1 per row instead of held in registers
__device__ __forceinline__ cd ldc_row(const double2* b, long e, long n, long i) {
  double x, y;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "l"(b + e * n + i));
  return cd{x, y};
}

// the 13 coefficient columns of one (node, z row) of the scattered terms (no direct term), as
// coef1d_row, from the W-weighted amplitudes (fin0 applied; shared memory, aw[(m 2 + br) 3 + q]
// [thread]) and the four branch phases g[m][br] (phase_cl(kz, z or z - d_obs) kx)
__device__ __forceinline__ void coef_row_scat(const CacheView& c, long k, const double2 (*aw)[128], const cd g[2][2],
                                              cd c0[5], cd c1[4], cd c2[4]) {
  const long n = c.n;
  const cd half_i{0.0, 0.5};
#pragma unroll
  for (int i = 0; i < 5; ++i) c0[i] = cd{0, 0};
#pragma unroll
  for (int i = 0; i < 4; ++i) { c1[i] = cd{0, 0}; c2[i] = cd{0, 0}; }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int br = 0; br < 2; ++br) {
      const cd ex = ldc_row(c.basis, (br == 0 ? 0 : 6) + m, n, k);
      const cd ey = ldc_row(c.basis, (br == 0 ? 2 : 8) + m, n, k);
      const cd ez = ldc_row(c.basis, (br == 0 ? 4 : 10) + m, n, k);
      const int e0 = (m * 2 + br) * 3;
      const double2 a0 = aw[e0][threadIdx.x], a1 = aw[e0 + 1][threadIdx.x], a2 = aw[e0 + 2][threadIdx.x];
      const cd ax = cd{a0.x, a0.y} * g[m][br], ay = cd{a1.x, a1.y} * g[m][br], az = cd{a2.x, a2.y} * g[m][br];
      c0[0] += half_i * (-(ax * ex) - ay * ey);
      c2[0] += half_i * (ax * ex - ay * ey);
      c0[1] += half_i * (-(ax * ey) + ay * ex);
      c2[1] += half_i * (ax * ey + ay * ex);
      c1[0] += ax * ez;
      c0[2] += half_i * (-(ay * ex) + ax * ey);
      c2[2] += half_i * (ay * ex + ax * ey);
      c0[3] += half_i * (-(ay * ey) - ax * ex);
      c2[3] += half_i * (ay * ey - ax * ex);
      c1[1] += ay * ez;
      c1[2] += az * ex;
      c1[3] += az * ey;
      c0[4] += cd{0.0, -1.0} * (az * ez);
    }
}

// rows z0..z1-1 of a node with the same-layer direct term (coef1d_row), out of line so that its
// registers and local arrays stay out of the scattered path
__device__ __noinline__ void coef_rows_direct(const Synth1DItem& it, long k, int z0, int z1) {
  const SynthParams& p = it.sp;
  const long n = p.c.n;
  const int nz = p.nz;
  const long cst = it.ldc;  // row stride of the coefficient columns
  float* C0 = it.C;
  float* C1 = it.C + (long)C1D_OFF1 * nz * cst;
  float* C2 = it.C + (long)C1D_OFF2 * nz * cst;
  cd Af[2][3], Ab[2][3];
  for (int m = 0; m < 2; ++m)
    for (int q = 0; q < 3; ++q) {
      Af[m][q] = ldc(it.amp, 3 * m + q, n, k);
      Ab[m][q] = ldc(it.amp, 6 + 3 * m + q, n, k);
    }
  for (int zi = z0; zi < z1; ++zi) {
    cd c0[5], c1[4], c2[4];
    coef1d_row(p, k, p.zo[zi], Af, Ab, c0, c1, c2);
    store_coef_row(C0, C1, C2, cst, k, zi, c0, c1, c2);
  }
}

// blocks of an item: ceil(n / 128) node blocks x ceil(nz / COEF1D_ZB_GROUP) height blocks,
// node block fastest. For
// the scattered terms at evenly spaced heights (it.dz != 0) the branch phases of a thread's
// consecutive rows follow by one complex product each, e^{i kz (z + dz)} = e^{i kz z} e^{i kz dz};
// a row whose exponent leaves phase_cl's range (or a step that overflows) takes phase_cl itself.
__global__ void __launch_bounds__(128, 3) k_coef1d_group(const Synth1DItem* __restrict__ items,
                                                      const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const Synth1DItem& it = items[i];
  const SynthParams& p = it.sp;
  const CacheView& c = p.c;
  const long n = c.n;
  const long nkb = (n + 127) / 128;
  const long b = blockIdx.x - first[i];
  const long k = (b % nkb) * 128 + threadIdx.x;
  if (k >= n) return;
  const int nz = p.nz;
  const long cst = it.ldc;  // row stride of the coefficient columns
  float* C0 = it.C;
  float* C1 = it.C + (long)C1D_OFF1 * nz * cst;
  float* C2 = it.C + (long)C1D_OFF2 * nz * cst;
  const int z0 = (int)(b / nkb) * COEF1D_ZB_GROUP;
  const int z1 = min(nz, z0 + COEF1D_ZB_GROUP);
  if (p.with_direct) {
    coef_rows_direct(it, k, z0, z1);
    return;
  }
  // the node's W-weighted amplitudes and its four kz in shared memory (read once per row and
  // branch; registers hold the row's accumulators and phases)
  __shared__ double2 aw[12][128];
  __shared__ double2 skz[4][128];
  const cd W = cd{0.0, 1.0 / (2.0 * 3.14159265358979323846)} * cd{c.wr[k], 0.0};
  const cd kx{c.kr[k], 0.0};
#pragma unroll
  for (int m = 0; m < 2; ++m) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const cd f = fin0(W * ldc(it.amp, 3 * m + q, n, k)), bk = fin0(W * ldc(it.amp, 6 + 3 * m + q, n, k));
      aw[(m * 2) * 3 + q][threadIdx.x] = make_double2(f.x, f.y);
      aw[(m * 2 + 1) * 3 + q][threadIdx.x] = make_double2(bk.x, bk.y);
    }
    skz[m * 2][threadIdx.x] = c.basis[(12L + m) * n + k];
    skz[m * 2 + 1][threadIdx.x] = c.basis[(14L + m) * n + k];
  }
  const double dz = it.dz;
  cd ph[2][2], step[2][2];
  bool have[2][2];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int br = 0; br < 2; ++br) {
      have[m][br] = false;
      ph[m][br] = cd{0, 0};
      const double2 q = skz[m * 2 + br][threadIdx.x];
      step[m][br] = dz != 0.0 ? cexp_call(-q.y * dz, q.x * dz) : cd{0, 0};
      if (!(dz != 0.0 && isfin(step[m][br]))) step[m][br] = cd{0, 0};
    }
  for (int zi = z0; zi < z1; ++zi) {
    const double zf = p.zo[zi], zb = zf - p.d_obs;
    cd g[2][2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int br = 0; br < 2; ++br) {
        const double2 q = skz[m * 2 + br][threadIdx.x];
        const double zz = br == 0 ? zf : zb;
        const double a = -q.y * zz, bb = q.x * zz;
        if (!isfinite(a) || !isfinite(bb) || a > 700.0 || a < -700.0) {
          ph[m][br] = cd{0, 0};
          have[m][br] = false;
        } else if (have[m][br] && (step[m][br].x != 0.0 || step[m][br].y != 0.0)) {
          ph[m][br] = ph[m][br] * step[m][br];
        } else {
          ph[m][br] = cexp_call(a, bb);
          have[m][br] = true;
        }
        g[m][br] = ph[m][br] * kx;
      }
    cd c0[5], c1[4], c2[4];
    coef_row_scat(c, k, aw, g, c0, c1, c2);
    store_coef_row(C0, C1, C2, cst, k, zi, c0, c1, c2);
  }
}

__global__ void __launch_bounds__(128, 4) k_reflect_sym_group(const Synth1DItem* __restrict__ items,
                                                           const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const long k = (long)(blockIdx.x - first[i]) * blockDim.x + threadIdx.x;
  if (k < items[i].sp.c.n) reflect_sym_body(items[i].sp, k, items[i].amp);
}
// node block fastest, as k_coef1d_group. Four CTAs per SM: 32 film stacks (325k nodes x 64 heights) 278 us, 287 us
// at three; in a group the fourth CTA hides more than its 128 bytes of spilled stores a thread cost, one
// stack by itself (k_coef_sym) is faster at three
__global__ void __launch_bounds__(128, 4) k_coef_sym_group(const Synth1DItem* __restrict__ items,
                                                           const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const Synth1DItem& it = items[i];
  const SynthParams& p = it.sp;
  const long nkb = (p.c.n + 127) / 128, b = blockIdx.x - first[i];
  const long k = (b % nkb) * 128 + threadIdx.x;
  if (k >= p.c.n) return;
  const int z0 = (int)(b / nkb) * COEF_SYM_ZB;
  float* C1 = it.C + (long)C1S_R0 * p.nz * it.ldc;
  coef_sym_rows(p, it.amp, k, z0, min(p.nz, z0 + COEF_SYM_ZB), it.dz, it.C, C1, C1 + (long)C1S_R1 * p.nz * it.ldc,
                it.ldc);
}

cudaError_t launch_reflect_coef_group(const Synth1DGroup& g, int stage, cudaStream_t s) {
  if (g.ni <= 0) return cudaSuccess;
  if (stage == 0 && g.grid[7] > 0) k_reflect_sym_group<<<(unsigned)g.grid[7], 128, 0, s>>>(g.it, g.first_rsym, g.ni);
  if (stage == 1 && g.grid[8] > 0) k_coef_sym_group<<<(unsigned)g.grid[8], 128, 0, s>>>(g.it, g.first_csym, g.ni);
  if (stage == 0 && g.grid[0] > 0) k_reflect2d_group<<<(unsigned)g.grid[0], 128, 0, s>>>(g.it, g.first_reflect, g.ni);
  if (stage == 1 && g.grid[1] > 0) k_coef1d_group<<<(unsigned)g.grid[1], 128, 0, s>>>(g.it, g.first_coef, g.ni);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(128) k_assemble1d_group(const Synth1DItem* __restrict__ items,
                                                          const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  assemble1d_body(items[i].a, blockIdx.x - first[i]);
}

cudaError_t launch_assemble1d_group(const Synth1DGroup& g, cudaStream_t s) {
  if (g.ni <= 0 || g.grid[5] <= 0) return cudaSuccess;
  k_assemble1d_group<<<(unsigned)g.grid[5], 128, 0, s>>>(g.it, g.first_asm, g.ni);
  return cudaGetLastError();
}

}  // namespace ytf

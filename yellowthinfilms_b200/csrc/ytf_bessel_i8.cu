// ytf_bessel_i8.cu -- the 1D Bessel synthesis contraction on the int8 tensor cores.
//
// closed_form_G for 1D caches (mod_ClosedFormField.jl:435-487) contracts, per Bessel order n,
//   P_n[r][c] = Σ_k J_n(k_k ρ_r) C_n[c][k]
// (C_n: the real and imaginary parts of the order's coefficient columns, k_coef_sym or k_coef1d_amp). Both
// operands are fixed point in three signed base-256 digits, as in the 2D lateral kernel:
//   J: X = rint(8355000 J / j_env(k_min ρ))   per (radius, node slice): |J_n| ≤ j_env
//   C: Y = rint(8355000 C / max|C|)   per (node slice, column)
// and the six digit products of weight ≥ 256² are summed exactly in INT32 in tensor memory.
// Unlike the lateral kernel, both operands are prepared once per launch as the exact shared-
// memory image of each 64-node stage (k_aimg_bessel3 evaluates J_n straight into digits; no
// FP64 table), so the contraction kernel only streams images: warp 0 issues the two bulk
// copies of a stage (one mbarrier, byte-counted), one thread of warp 1 issues the 12 MMAs
// (6 digit products x 2 K-halves; M=128 radii, N ≤ 160 columns, K=32), warps 2-5 read the
// accumulators at the end.
// INT32 headroom: |level-2 sum| ≤ (127·128 + 128·128 + 128·127) K ≤ 48896 · 16384 < 2^30.
#include "ytf_complex.cuh"
#include "ytf_kernels.h"
#include "ytf_bessel.cuh"
#include "ytf_tcgen05.cuh"

namespace ytf {

constexpr int BI_M = 128;
constexpr int BI_NODES = 64;  // nodes per stage: one byte each, 64-byte rows (2 MMAs of K = 32)
constexpr int BI_STAGES = 4;
constexpr int BI_THREADS = 192;
constexpr int BI_ACC_STRIDE = 160;
constexpr int BI_TMEM_COLS = 512;
constexpr long BI_WAIT_LIMIT = 1L << 22;  // polls of the drain waits (the pipeline waits: p.wait_limit)
constexpr double BI_SCALE = 8355000.0;

size_t bessel_i8_stage_bytes_a() { return 3ul * BI_M * 64; }
size_t bessel_i8_stage_bytes_b(int Np) { return 3ul * (size_t)Np * 64; }
size_t bessel_i8_smem(int Np) {
  return (size_t)BI_STAGES * (bessel_i8_stage_bytes_a() + bessel_i8_stage_bytes_b(Np)) + 8 * BI_ACC_STRIDE + 128;
}
int bessel_i8_ctile(int N) {
  int nt = (N + 159) / 160;
  return (N + nt - 1) / nt;
}

// J_2 from J_0, J_1 at x >= 0, y = 1 / x: its power series below x = 1 (A&S 9.1.10; exact 0 at x = 0;
// 9 terms, the first left out below 1e-18) and the three-term recurrence above (A&S 9.1.27)
__device__ __forceinline__ double j2_from(double x, double y, double J0, double J1) {
  if (x < 1.0) {
    // (h2 / 2) Σ_m (-h2)^m 2 / (m! (m + 2)!), h2 = x² / 4
    const double h2 = 0.25 * x * x;
    double s = 1.0 / (40320.0 * 1814400.0);
    s = fma(s, h2, -1.0 / (5040.0 * 181440.0));
    s = fma(s, h2, 1.0 / (720.0 * 20160.0));
    s = fma(s, h2, -1.0 / (120.0 * 2520.0));
    s = fma(s, h2, 1.0 / (24.0 * 360.0));
    s = fma(s, h2, -1.0 / (6.0 * 60.0));
    s = fma(s, h2, 1.0 / (2.0 * 12.0));
    s = fma(s, h2, -1.0 / 3.0);
    s = fma(s, h2, 1.0);
    return 0.5 * h2 * s;
  }
  return fma(2.0 * y, J1, -J0);
}

// J_0(x), J_1(x) for 0 <= x < 25 from the Taylor rows (tab: JTAB, or a copy of it in shared memory): one
// Horner pass for the value and the derivative, 31 FP64 operations for both orders, |error| <= 2e-16.
// The math library's j0 and j1 take their own argument ranges apart in every warp: 4096 radii x 65536
// nodes, 64% of them below 25: 3183 us with them, 1395 us in the present image kernel.
__device__ __forceinline__ void j01_small(double x, const double* __restrict__ tab, double& J0, double& J1) {
  const int i = min(max((int)x, 0), JTAB_N - 1);
  const double d = x - ((double)i + 0.5);
  const double* c = tab + i * JTAB_M;
  double p = c[JTAB_M - 1], q = 0.0;
#pragma unroll
  for (int m = JTAB_M - 2; m >= 0; --m) {
    q = fma(q, d, p);
    p = fma(p, d, c[m]);
  }
  J0 = p;
  J1 = -q;
}

// J_0(x) and J_1(x) for x >= 25 (absolute error below 1e-12): Hankel's asymptotic expansions
// (A&S 9.2.5, 9.2.9, 9.2.10), J_n(x) = sqrt(2 / (π x)) (P_n cos χ_n - Q_n sin χ_n) with
// χ_n = x - (2n + 1) π / 4, five terms each of P_n and Q_n in y = 1/x (the coefficient of y^m
// is ±a_m / 8^m, a_m = Π_{j<=m} (4n² - (2j - 1)²) / m!). Both orders share one phase
// (χ_1 = χ_0 - π/2): χ_0 = r + n π/2, |r| <= π/4, by a Cody-Waite reduction of x by (n + 1/2) π/2 (a
// three-part constant whose first two parts carry 33 bits, so its products are exact for n < 2^19)
// and Taylor polynomials for sin r and cos r (to r^17 and r^18). The library's j0 and j1 evaluate each
// order with its own phase.
constexpr double J_ASYM_MIN = 25.0;
// y = 1 / x, a = sqrt(2 / (π x)) (products of per-node and per-radius factors in the image kernel)
__device__ __forceinline__ void j01_large(double x, double y, double a, double& J0, double& J1) {
  const double y2 = y * y;
  const double p0 = fma(fma(fma(fma(6.074042001273483, y2, -0.5725014209747314), y2, 0.112152099609375), y2,
                            -0.0703125), y2, 1.0);
  const double q0 = y * fma(fma(fma(fma(-24.380529699556064, y2, 1.7277275025844574), y2, -0.22710800170898438), y2,
                                0.0732421875), y2, -0.125);
  const double p1 = fma(fma(fma(fma(-6.883914268109947, y2, 0.6765925884246826), y2, -0.144195556640625), y2,
                            0.1171875), y2, 1.0);
  const double q1 = y * fma(fma(fma(fma(27.248827311268542, y2, -1.993531733751297), y2, 0.2775764465332031), y2,
                                -0.1025390625), y2, 0.375);
  // x - π/4 = n π/2 + r, |r| <= π/4: n = floor(2 x / π), rounded down onto the whole numbers at 1.5 2^52,
  // whose low bits hold it
  const double nm = __fma_rd(x, 0.6366197723675814, 6755399441055744.0);
  const double m = (nm - 6755399441055744.0) + 0.5;
  double r = fma(-m, 1.5707963267341256, x);
  r = fma(-m, 6.077100506303966e-11, r);
  r = fma(-m, 2.0222662487959506e-21, r);
  const double r2 = r * r;
  double sr = fma(fma(fma(fma(fma(fma(fma(2.8114572543455206e-15, r2, -7.647163731819816e-13), r2,
                                          1.6059043836821613e-10), r2, -2.505210838544172e-08), r2,
                                  2.7557319223985893e-06), r2, -0.0001984126984126984), r2, 0.008333333333333333), r2,
                  -0.16666666666666666);
  sr = fma(r * r2, sr, r);
  double cr = fma(fma(fma(fma(fma(fma(fma(fma(-1.5619206968586225e-16, r2, 4.779477332387385e-14), r2,
                                          -1.1470745597729725e-11), r2, 2.08767569878681e-09), r2,
                                  -2.755731922398589e-07), r2, 2.48015873015873e-05), r2, -0.001388888888888889), r2,
                  0.041666666666666664), r2, -0.5);
  cr = fma(r2, cr, 1.0);
  // quadrant n: swap for odd n, signs from bit 1 of n (sine) and of n + 1 (cosine)
  const int q = __double2loint(nm);
  const double ss = q & 1 ? cr : sr, cc = q & 1 ? sr : cr;
  const double s0 = __hiloint2double(__double2hiint(ss) ^ ((q & 2) << 30), __double2loint(ss));
  const double c0 = __hiloint2double(__double2hiint(cc) ^ (((q + 1) & 2) << 30), __double2loint(cc));
  J0 = a * (p0 * c0 - q0 * s0);
  J1 = a * (p1 * s0 + q1 * c0);
}
// J_0, J_1 as the int8x3 J images take them: the asymptotic pair from x = 25, the Taylor rows below; J_1
// below x = 1 from its series, which agrees with the rows to 1e-16 of 1 and keeps its relative accuracy down to 0
__device__ __forceinline__ void j01_real(double x, double& J0, double& J1) {
  const double ax = fabs(x);
  if (ax >= J_ASYM_MIN) {
    const double y = 1.0 / ax;
    j01_large(ax, y, 0.7978845608028654 * sqrt(y), J0, J1);
  } else {
    j01_small(ax, JTAB, J0, J1);
    if (ax < 1.0) J1 = 0.5 * ax * bessel_series_unit<1>(0.25 * x * x);
  }
  if (x < 0) J1 = -J1;  // J_1 is odd
}

__global__ void k_bessel_j01(const double* __restrict__ x, long n, double* __restrict__ J0, double* __restrict__ J1) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a, b;
  j01_real(x[i], a, b);
  J0[i] = a;
  J1[i] = b;
}
cudaError_t launch_bessel_j01(const double* x, long n, double* J0, double* J1, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_bessel_j01<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, n, J0, J1);
  return cudaGetLastError();
}

// |J_n(x)| <= j_env(x) = min(1, 0.9 / sqrt(x)) for n = 0, 1, 2 and x >= 0 (the suprema of
// sqrt(x) |J_n(x)| are 0.798, 0.825, 0.868 for n = 0, 1, 2); non-increasing, so j_env(k_min ρ)
// bounds J_n(k ρ) over a node slice whose smallest node is k_min. The J digits of a (radius,
// slice) are fixed point relative to it, so far radii keep their 24 bits.
__device__ __forceinline__ double j_env(double x) { return x > 0.81 ? 0.9 / sqrt(x) : 1.0; }

// the smallest node of every slice: one block of 256 threads per slice (kmin[z])
__device__ __forceinline__ void slice_kmin_body(const double* kr, long K, long kchunk, int z, double* kmin) {
  __shared__ double red[256];
  const long k0 = (long)z * kchunk, k1 = min(K, k0 + kchunk);
  double m = INFINITY;
  for (long k = k0 + threadIdx.x; k < k1; k += blockDim.x) m = fmin(m, kr[k]);
  red[threadIdx.x] = m;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] = fmin(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) kmin[z] = isfinite(red[0]) ? red[0] : 0.0;
}
__global__ void __launch_bounds__(256) k_slice_kmin(const double* kr, long K, long kchunk, double* kmin) {
  slice_kmin_body(kr, K, kchunk, blockIdx.x, kmin);
}
cudaError_t launch_slice_kmin(const double* kr, long K, long kchunk, int nchunk, double* kmin, cudaStream_t s) {
  if (nchunk <= 0) return cudaSuccess;
  k_slice_kmin<<<(unsigned)nchunk, 256, 0, s>>>(kr, K, kchunk, kmin);
  return cudaGetLastError();
}

__device__ __forceinline__ double col_scale(unsigned long long bits) {
  const double m = __longlong_as_double((long long)bits);
  return (m > 0.0 && isfinite(m)) ? BI_SCALE / m : 0.0;
}

// entries c[k .. k + 3] (k a multiple of 4, c's rows on 16 bytes), zero at k >= K
__device__ __forceinline__ float4 load4(const float* c, long k, long K) {
  if (k + 4 <= K) return __ldg(reinterpret_cast<const float4*>(c + k));
  return make_float4(k < K ? c[k] : 0.0f, k + 1 < K ? c[k + 1] : 0.0f, k + 2 < K ? c[k + 2] : 0.0f, 0.0f);
}

// the coefficient digit images and their (slice, column) maxima: one block per (column tile, 8-slot row
// group, node slice), its warps taking the slice's 64-node stages in turn, lane (r8, t) = (lane >> 2,
// lane & 3) column slot 8 rg + r8 and nodes 16 i + 4 t .. + 3, i < 4, of a stage: every load takes 64
// consecutive bytes of eight columns, every store one whole 128-byte line of a digit plane. A first pass
// reduces max |C| (IEEE bits into colmax: a non-finite entry counts as Inf), a second reads the same
// bytes again (from L2) and writes the digits. Blocks: ntile_n x (Np / 8) x nchunk.
// Bound by the loads in flight: two stages' in the first pass, the next stage's in the second. 65536 nodes x
// 2560 columns 367 us with 64 bytes of a column per thread (16 lines touched by each load, one stage in
// flight, blocks of 256) and the digits by conversions and shifts; 303 us. 32 film stacks x 64 heights in
// 4096-node slices (237M values) 349 us; 335-347 us.
__device__ __forceinline__ void bimg_slice_body(const BesselI8& p, long b) {
  __shared__ float wmax[32][8];
  const int tid = threadIdx.x, lane = tid & 31, r8 = lane >> 2, t4 = 4 * (lane & 3);
  const int warp = tid >> 5, nwarp = blockDim.x >> 5;
  const int rgroups = p.Np / 8;
  const int rg = (int)(b % rgroups);
  const long rest = b / rgroups;
  const int z = (int)(rest % p.nchunk);
  const int ct = (int)(rest / p.nchunk);
  const int slot = rg * 8 + r8;
  const int col = ct * p.ctile + slot;
  const bool cv = slot < p.ctile && col < p.N;
  const float* c = p.C + (long)(cv ? col : 0) * p.ldc;
  const long K = cv ? p.K : 0, kbase = (long)z * p.kchunk + t4;
  const int nstage = (int)(p.kchunk / BI_NODES);
  int mi = 0;  // |C| orders as its bits; NaN above Inf
  for (int s = warp; s < nstage; s += 2 * nwarp) {  // two stages' loads in flight
    float4 f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int st = s + (i >> 2) * nwarp;
      f[i] = load4(c, kbase + 64L * st + 16 * (i & 3), st < nstage ? K : 0);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mi = max(max(mi, __float_as_int(f[i].x) & 0x7fffffff), __float_as_int(f[i].y) & 0x7fffffff);
      mi = max(max(mi, __float_as_int(f[i].z) & 0x7fffffff), __float_as_int(f[i].w) & 0x7fffffff);
    }
  }
  // the four lanes of a slot, then the block's warps
  float m = __int_as_float(min(mi, 0x7f800000));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (t4 == 0) wmax[warp][r8] = m;
  __syncthreads();
  float mm = wmax[0][r8];
  for (int w = 1; w < nwarp; ++w) mm = fmaxf(mm, wmax[w][r8]);
  const unsigned long long bits = (unsigned long long)__double_as_longlong((double)mm);
  if (warp == 0 && t4 == 0 && cv) p.colmax[(long)z * p.N + col] = bits;
  const double sB = cv ? col_scale(bits) : 0.0;
  const size_t plane = (size_t)p.Np * 64, sbytes = 3 * plane;
  uint8_t* base = p.Bimg + ((size_t)ct * p.nchunk + z) * nstage * sbytes + t4;
  float4 f[4], nx[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) nx[i] = load4(c, kbase + 64L * warp + 16 * i, warp < nstage ? K : 0);
  for (int s = warp; s < nstage; s += nwarp) {
    const int s1 = s + nwarp;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[i] = nx[i];
      nx[i] = load4(c, kbase + 64L * s1 + 16 * i, s1 < nstage ? K : 0);
    }
    uint8_t* blk = base + (size_t)s * sbytes;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t u[4] = {fixed_bits((double)f[i].x, sB),
                             fixed_bits((double)f[i].y, sB),
                             fixed_bits((double)f[i].z, sB),
                             fixed_bits((double)f[i].w, sB)};
      uint32_t d0, d1, d2;
      digit_words(u, d0, d1, d2);
      uint8_t* dst = blk + plane_off(slot, 16 * i);
      *reinterpret_cast<uint32_t*>(dst) = d0;
      *reinterpret_cast<uint32_t*>(dst + plane) = d1;
      *reinterpret_cast<uint32_t*>(dst + 2 * plane) = d2;
    }
  }
}

// ------------------------------------------------------------------------------------
// The J_n(k ρ) digit images of all three orders: J_0 and J_1 once per (ρ, k), J_2 from them. A block
// takes one 64-node stage of p.arows rows of a radius tile: thread (w, r) = (tid & 15, tid >> 4) nodes
// 4 w .. 4 w + 3 of rows r, r + 16, ..., so that 1/k and 1/sqrt(k) are formed once per thread, 1/ρ,
// sqrt(2/(π ρ)) and the row's digit scale once per row, and a pair needs no division and no root. Where
// a warp's pairs all lie on one side of x = 25 a thread's four run side by side. The
// fixed-point value comes from one FMA: v sA + 1.5 2^52 + 0x808080 holds rint(v sA) + 0x808080 in its
// low word, whose bytes are the three digits with their sign bits flipped; four nodes' words transpose
// into one word per digit plane by byte permutes.
//   Bound: the FP64 pipe (59% busy; about 40 operations per pair below x = 25 and 60 above) and the wait
// between dependent ones. 325k nodes x 256 radii: 491 us; with 64-bit index divisions, library j0 and
// j1, a division and a root per pair and FP64-to-integer conversions, 1363 us; this form with 32-row
// blocks and one pair after the other, 806 us.
// ------------------------------------------------------------------------------------

// rows per block: a whole tile (the per-thread reciprocals then serve 32 pairs) once the stages alone
// give each SM eight blocks, a quarter of it below
int bessel_i8_arows(long stages) { return stages >= 8 * 148 ? BI_M : BI_M / 4; }
long bessel_i8_aimg_blocks(const BesselI8& p) {
  return (long)p.ntile_m * (BI_M / p.arows) * p.nchunk * (p.kchunk / BI_NODES);
}

__device__ __forceinline__ void aimg_bessel3_body(const BesselI8& p, long b, uint8_t* __restrict__ A0,
                                                  uint8_t* __restrict__ A1, uint8_t* __restrict__ A2) {
  __shared__ double tab[JTAB_N * JTAB_M];
  __shared__ double rho_s[BI_M], rrho_s[BI_M], srho_s[BI_M], scale_s[BI_M];
  const int tid = threadIdx.x;
  const int nst = (int)(p.kchunk / BI_NODES);
  const int arows = p.arows;
  // stage fastest, then the slice, the row group, the radius tile
  const unsigned ub = (unsigned)b;
  const int s = (int)(ub % (unsigned)nst);
  const unsigned u1 = ub / (unsigned)nst;
  const int z = (int)(u1 % (unsigned)p.nchunk);
  const unsigned u2 = u1 / (unsigned)p.nchunk;
  const unsigned rgroups = (unsigned)(BI_M / arows);
  const int rb = (int)(u2 % rgroups), mt = (int)(u2 / rgroups);
  for (int i = tid; i < JTAB_N * JTAB_M; i += 256) tab[i] = JTAB[i];
  if (tid < arows) {
    const int r = mt * BI_M + rb * arows + tid;
    const double rho = r < p.M ? p.rho[r] : 0.0, ar = fabs(rho);
    rho_s[tid] = rho;
    rrho_s[tid] = 1.0 / ar;
    srho_s[tid] = 0.7978845608028654 * sqrt(1.0 / ar);
    scale_s[tid] = BI_SCALE / j_env(p.kmin[z] * rho);
  }
  const int w = tid & 15, rr = tid >> 4;
  const long k0 = (long)z * p.kchunk + (long)s * BI_NODES + 4 * w;
  double kv[4], rk[4], sk[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    kv[h] = k0 + h < p.K ? p.kr[k0 + h] : 0.0;
    rk[h] = 1.0 / fabs(kv[h]);
    sk[h] = sqrt(rk[h]);
  }
  __syncthreads();
  const size_t off = (((size_t)mt * p.nchunk + z) * nst + s) * (3ul * BI_M * 64);
  uint8_t* out[3] = {A0 + off, A1 + off, A2 + off};
#pragma unroll 1
  for (int i = 0; i < arows / 16; ++i) {
    const int lr = rr + 16 * i, row = rb * arows + lr;
    const bool rv = mt * BI_M + row < p.M;
    const double rho = rho_s[lr], rrho = rrho_s[lr], srho = srho_s[lr], sA = scale_s[lr];
    double x[4], v0[4], v1[4], v2[4];
    bool small = true, large = true, over1 = true;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      x[h] = fabs(kv[h] * rho);
      small = small && !(x[h] >= J_ASYM_MIN);
      large = large && x[h] >= J_ASYM_MIN;
      over1 = over1 && x[h] >= 1.0;
    }
    if (__all_sync(0xffffffffu, large)) {
#pragma unroll
      for (int h = 0; h < 4; ++h) j01_large(x[h], rk[h] * rrho, sk[h] * srho, v0[h], v1[h]);
    } else if (__all_sync(0xffffffffu, small)) {
#pragma unroll
      for (int h = 0; h < 4; ++h) j01_small(x[h], tab, v0[h], v1[h]);
    } else {
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        if (x[h] >= J_ASYM_MIN) j01_large(x[h], rk[h] * rrho, sk[h] * srho, v0[h], v1[h]);
        else j01_small(x[h], tab, v0[h], v1[h]);
      }
    }
    if (__all_sync(0xffffffffu, over1)) {
#pragma unroll
      for (int h = 0; h < 4; ++h) v2[h] = fma(2.0 * (rk[h] * rrho), v1[h], -v0[h]);
    } else {
#pragma unroll
      for (int h = 0; h < 4; ++h) v2[h] = j2_from(x[h], rk[h] * rrho, v0[h], v1[h]);
    }
    uint32_t U[3][4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const bool live = rv && k0 + h < p.K;
      const double s1 = kv[h] * rho < 0 ? -sA : sA;  // J_1 is odd
      U[0][h] = (uint32_t)__double2loint(fma(live ? v0[h] : 0.0, sA, AI_MAGIC));
      U[1][h] = (uint32_t)__double2loint(fma(live ? v1[h] : 0.0, s1, AI_MAGIC));
      U[2][h] = (uint32_t)__double2loint(fma(live ? v2[h] : 0.0, sA, AI_MAGIC));
    }
    const uint32_t at = plane_off(row, 4 * w);
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      uint32_t d0, d1, d2;
      digit_words(U[o], d0, d1, d2);
      uint8_t* dst = out[o] + at;
      *reinterpret_cast<uint32_t*>(dst) = d0;
      *reinterpret_cast<uint32_t*>(dst + BI_M * 64) = d1;
      *reinterpret_cast<uint32_t*>(dst + 2 * BI_M * 64) = d2;
    }
  }
}
__global__ void __launch_bounds__(256, 3) k_aimg_bessel3(const __grid_constant__ BesselI8 p, uint8_t* __restrict__ A0,
                                                      uint8_t* __restrict__ A1, uint8_t* __restrict__ A2) {
  aimg_bessel3_body(p, blockIdx.x, A0, A1, A2);
}

cudaError_t launch_bessel_i8_aimg3(const BesselI8& p, uint8_t* A0, uint8_t* A1, uint8_t* A2, cudaStream_t s) {
  if (p.M <= 0 || p.K <= 0) return cudaSuccess;
  k_aimg_bessel3<<<(unsigned)bessel_i8_aimg_blocks(p), 256, 0, s>>>(p, A0, A1, A2);
  return cudaGetLastError();
}

// a row's digit scale from its slice maximum
__device__ __forceinline__ double row_scale(double m) { return m > 0.0 && isfinite(m) ? m : 1.0; }

struct BiShared {
  double fac[BI_ACC_STRIDE];  // per column: what one unit of the combined digits is worth
  uint64_t full[BI_STAGES], empty[BI_STAGES], done;
  uint32_t tmem;
  int abort_flag;
};

__device__ __forceinline__ bool bi_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned* err,
                                        long limit) {
  for (long it = 0; it < limit; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255 && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicOr(err, 1u);
  return false;
}
__device__ __forceinline__ void bi_drain_wait(uint32_t bar, uint32_t parity) {
  for (long it = 0; it < BI_WAIT_LIMIT; ++it)
    if (mbar_try(bar, parity)) return;
}

// one CTA's (radius tile mt, column tile ct, node slice z) contraction; every thread calls it
__device__ __forceinline__ void gemm_i8_img_body(const BesselI8& p, int mt, int ct, int z, uint8_t* smem) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = ct * p.ctile;
  const int nct = min(p.ctile, p.N - c0);
  const long k0 = (long)z * p.kchunk, k1 = min(p.K, k0 + p.kchunk);
  const int nst = k1 > k0 ? (int)((k1 - k0 + BI_NODES - 1) / BI_NODES) : 0;
  const long nstage_chunk = p.kchunk / BI_NODES;
  const uint32_t planeA = BI_M * 64u, planeB = (uint32_t)p.Np * 64u;
  const uint32_t stageA = 3u * planeA, stageB = 3u * planeB;
  uint8_t* smA = smem;
  uint8_t* smB = smem + BI_STAGES * stageA;
  BiShared* sh = reinterpret_cast<BiShared*>(smB + BI_STAGES * stageB);
  volatile int* abort_flag = &sh->abort_flag;
  if (tid == 0) {
    for (int s = 0; s < BI_STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    mbar_init(smem_u32(&sh->done), 1);
    sh->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem)),
                 "r"(BI_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;

  if (warp == 0) {
    if (lane == 0) {
      const uint8_t* gA = p.Aimg + ((size_t)mt * p.nchunk + z) * nstage_chunk * stageA;
      const uint8_t* gB = p.Bimg + ((size_t)ct * p.nchunk + z) * nstage_chunk * stageB;
      int issued = 0;
      for (int s = 0; s < nst; ++s) {
        const int slot = s % BI_STAGES;
        if (s >= BI_STAGES && !bi_wait(smem_u32(&sh->empty[slot]), ((s / BI_STAGES) - 1) & 1, abort_flag, p.err, p.wait_limit))
          break;
        const uint32_t bar = smem_u32(&sh->full[slot]);
        mbar_arrive_tx(bar, stageA + stageB);
        bulk_g2s(smem_u32(smA + slot * stageA), gA + (size_t)s * stageA, stageA, bar);
        bulk_g2s(smem_u32(smB + slot * stageB), gB + (size_t)s * stageB, stageB, bar);
        issued = s + 1;
      }
      for (int s = max(0, issued - BI_STAGES); s < issued; ++s)
        bi_drain_wait(smem_u32(&sh->full[s % BI_STAGES]), (s / BI_STAGES) & 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc =
          (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.Np >> 3) << 17) | ((uint32_t)(BI_M >> 4) << 24);
      const int pa[6] = {0, 0, 1, 0, 1, 2}, pb[6] = {0, 1, 0, 2, 1, 0};
      for (int s = 0; s < nst; ++s) {
        const int slot = s % BI_STAGES;
        if (!bi_wait(smem_u32(&sh->full[slot]), (s / BI_STAGES) & 1, abort_flag, p.err, p.wait_limit)) break;
        tc_fence_after();
        const uint32_t a0 = smem_u32(smA + slot * stageA), b0 = smem_u32(smB + slot * stageB);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int pr = 0; pr < 6; ++pr) {
            const uint64_t ad = umma_desc(a0 + pa[pr] * planeA + t * 256u);
            const uint64_t bd = umma_desc(b0 + pb[pr] * planeB + t * 256u);
            const bool first = s == 0 && t == 0 && (pr == 0 || pr == 1 || pr == 3);
            asm volatile(
                "{\n\t.reg .pred PD;\n\t"
                "setp.ne.b32 PD, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, PD;\n\t}" ::"r"(
                    tmem + (uint32_t)((pa[pr] + pb[pr]) * BI_ACC_STRIDE)),
                "l"(ad), "l"(bd), "r"(idesc), "r"(first ? 0u : 1u)
                : "memory");
          }
        tc_commit(smem_u32(&sh->empty[slot]));
      }
      tc_commit(smem_u32(&sh->done));
      if (*abort_flag) bi_drain_wait(smem_u32(&sh->done), 0);
    }
  } else {
    // epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. +31 (rows of the radius tile). The
    // columns' factors are formed once per CTA while the MMAs run: two FP64 divisions per value in the
    // drain took more than the MMAs of a short slice (440 CTAs of 3 stages each: 115 -> 44 us; 32 film
    // stacks 466 -> 310 us; 4096 radii x 256 heights 2.95 -> 2.66 ms)
    const unsigned long long* cmax = p.colmax + (long)z * p.N;
    for (int c = tid - 64; c < nct; c += 128) {
      const unsigned long long bits = cmax[c0 + c];
      const double m = __longlong_as_double((long long)bits);
      sh->fac[c] = !isfinite(m) ? __longlong_as_double(0x7ff8000000000000LL) : m > 0.0 ? 65536.0 / (BI_SCALE * col_scale(bits)) : 0.0;
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    bool ok = bi_wait(smem_u32(&sh->done), 0, abort_flag, p.err, p.wait_limit);
    ok = __all_sync(0xffffffffu, ok) && !*abort_flag;
    if (ok && nst > 0) {
      tc_fence_after();
      const int q = warp & 3;
      const uint32_t lanebase = (uint32_t)(32 * q) << 16;
      const int r = mt * BI_M + 32 * q + lane;
      const double eA = r >= p.M ? 1.0 : p.rowscale ? row_scale(p.rowscale[(long)z * p.M + r])
                                                     : j_env(p.kmin[z] * p.rho[r]);  // the row's J digit scale
      double* out = p.partial + (long)z * p.N * p.M;
      for (int e0 = 0; e0 < p.Np; e0 += 8) {
        uint32_t v0[8], v1[8], v2[8];
        tmem_ld8(tmem + lanebase + e0, v0);
        tmem_ld8(tmem + lanebase + BI_ACC_STRIDE + e0, v1);
        tmem_ld8(tmem + lanebase + 2 * BI_ACC_STRIDE + e0, v2);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int cl = e0 + e;
          if (cl < nct && r < p.M) {
            const long long v = (long long)(int)v0[e] * 65536 + (long long)(int)v1[e] * 256 + (long long)(int)v2[e];
            out[(long)(c0 + cl) * p.M + r] = (double)v * sh->fac[cl] * eA;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    // after a timeout the epilogue may have stopped waiting for `done` while MMAs still run:
    // the MMA thread has committed `done` (it is past its loop), so wait for it before the
    // tensor memory is released
    if (*abort_flag && lane == 0) bi_drain_wait(smem_u32(&sh->done), 0);
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BI_TMEM_COLS) : "memory");
  }
}
// up to six entries by value; entry i's blocks start at first[i]
struct BesselI8Set {
  int n;
  long first[6];
  BesselI8 e[6];
};
__global__ void __launch_bounds__(BI_THREADS, 1) k_gemm_i8_img(const __grid_constant__ BesselI8Set set) {
  extern __shared__ __align__(1024) uint8_t smem[];
  int i = 0;
  while (i + 1 < set.n && set.first[i + 1] <= (long)blockIdx.x) ++i;
  const BesselI8& p = set.e[i];
  const long b = blockIdx.x - set.first[i];
  const int mt = (int)(b % p.ntile_m);
  const long rest = b / p.ntile_m;
  gemm_i8_img_body(p, mt, (int)(rest % p.ntile_n), (int)(rest / p.ntile_n), smem);
}
__global__ void __launch_bounds__(1024) k_bimg_real(const __grid_constant__ BesselI8Set set) {
  int i = 0;
  while (i + 1 < set.n && set.first[i + 1] <= (long)blockIdx.x) ++i;
  bimg_slice_body(set.e[i], blockIdx.x - set.first[i]);
}

// The digits of Re and Im J_o relative to the row's slice maximum. One warp per (64-node stage, eight rows,
// image), lane (r8, t) = (lane >> 2, lane & 3) row 8 blockIdx.y + r8 and nodes 16 i + 4 t .. + 3, i < 4: loads
// of 128 consecutive bytes per row, stores of whole 128-byte lines of a digit plane. Grid: x = stages (8 per
// block), y = row groups, z = image (2 o + part).
// Bound by memory: 256 rows x 4096 nodes x 6 tables (50 MB read, 19 MB written) 21.2 us with one 4-node word
// per thread (five 64-bit index divisions and one FP64 division each); 12.0 us.
struct Img6 {
  uint8_t* p[6];
};
__global__ void __launch_bounds__(256) k_jtab_img(BesselI8 p, const double* __restrict__ J,
                                                  const double* __restrict__ rs, Img6 img) {
  const int lane = threadIdx.x & 31, r8 = lane >> 2, t4 = 4 * (lane & 3);
  const unsigned nstage = (unsigned)(p.kchunk / BI_NODES);
  const unsigned st = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (st >= nstage * (unsigned)p.nchunk) return;
  const int z = (int)(st / nstage), s = (int)(st - z * nstage), im = blockIdx.z;
  const int r = 8 * blockIdx.y + r8, mt = r / BI_M, row = r % BI_M;
  const bool rv = r < p.M;
  const double sA = rv ? BI_SCALE / row_scale(rs[((long)(im / 2) * p.nchunk + z) * p.M + r]) : 0.0;
  const double* tab = J + (long)im * p.M * p.K + (long)(rv ? r : 0) * p.K;
  const long k0 = (long)z * p.kchunk + (long)s * BI_NODES + t4;
  double v[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 4; ++h) v[i][h] = rv && k0 + 16 * i + h < p.K ? __ldg(tab + k0 + 16 * i + h) : 0.0;
  uint8_t* blk = img.p[im] + (((size_t)mt * p.nchunk + z) * nstage + s) * (3ul * BI_M * 64) + t4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t u[4], w[3];
#pragma unroll
    for (int h = 0; h < 4; ++h) u[h] = (uint32_t)__double2int_rn(v[i][h] * sA) + 0x808080u;  // digits 0 for a NaN
    digit_words(u, w[0], w[1], w[2]);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
      *reinterpret_cast<uint32_t*>(blk + (size_t)pl * BI_M * 64 + plane_off(row, 16 * i)) = w[pl];
  }
}

cudaError_t launch_jtable_images(const BesselI8& bp, const double* Jtab, const double* rowscale, uint8_t* const img[6],
                                 cudaStream_t s) {
  if (bp.M <= 0 || bp.K <= 0) return cudaSuccess;
  const long stages = (long)bp.nchunk * (bp.kchunk / BI_NODES);
  Img6 im6;
  for (int i = 0; i < 6; ++i) im6.p[i] = img[i];
  k_jtab_img<<<dim3((unsigned)((stages + 7) / 8), (unsigned)(bp.ntile_m * BI_M / 8), 6), 256, 0, s>>>(bp, Jtab, rowscale, im6);
  return cudaGetLastError();
}

static bool entry_ok(const BesselI8& p) {
  return (p.kmin || p.rowscale) && p.kchunk % BI_NODES == 0 && p.kchunk <= 16384 && p.Np % 16 == 0 &&
         p.Np <= BI_ACC_STRIDE && p.Np >= p.ctile && (long)p.nchunk * p.kchunk >= p.K && p.ldc % 4 == 0;
}

// threads of a block of the coefficient images (see bimg_slice_body). Long slices: the resident blocks'
// slices, 32 bytes per node each, have to stay in L2 between the two passes (16384 nodes: 300 us at
// 1024 threads, 360 us at 256); short ones: no warp without a stage (192 nodes: 10.2 us at 128, 14.5 us at
// 256 threads).
static unsigned bimg_threads(long kchunk) {
  return kchunk > 10000 ? 1024 : kchunk > 5000 ? 512 : kchunk > 512 ? 256 : 128;
}

cudaError_t launch_bimg(const BesselI8* e, int n, cudaStream_t s) {
  BesselI8Set set;
  set.n = n;
  long blocks = 0;
  for (int i = 0; i < n; ++i) {
    if (!entry_ok(e[i])) return cudaErrorInvalidValue;
    set.e[i] = e[i];
    set.first[i] = blocks;
    blocks += (long)e[i].ntile_n * (e[i].Np / 8) * e[i].nchunk;
  }
  if (blocks <= 0) return cudaSuccess;
  k_bimg_real<<<(unsigned)blocks, bimg_threads(e[0].kchunk), 0, s>>>(set);
  return cudaGetLastError();
}

cudaError_t launch_gemm_i8(const BesselI8* e, int n, cudaStream_t s) {
  BesselI8Set set;
  set.n = n;
  long blocks = 0;
  int Np = 0;
  for (int i = 0; i < n; ++i) {
    if (!entry_ok(e[i])) return cudaErrorInvalidValue;
    set.e[i] = e[i];
    set.first[i] = blocks;
    blocks += (long)e[i].ntile_m * e[i].ntile_n * e[i].nchunk;
    Np = e[i].Np > Np ? e[i].Np : Np;
  }
  if (blocks <= 0) return cudaSuccess;
  const size_t sm = bessel_i8_smem(Np);
  cudaError_t err = cudaFuncSetAttribute(k_gemm_i8_img, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (err != cudaSuccess) return err;
  k_gemm_i8_img<<<(unsigned)blocks, BI_THREADS, sm, s>>>(set);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Grouped launches: every (item, order) entry of a group in one grid per stage. Entry
// e = 3 i + o holds item i's order-o parameters; its J_n images share item i's node slicing
// (bp[3 i] gives the layout), so one Bessel evaluation per (ρ, k) serves the three orders.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 3) k_aimg_bessel3_group(const BesselI8* __restrict__ bp, const long* __restrict__ first,
                                                          int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const BesselI8& p = bp[3 * i];
  aimg_bessel3_body(p, (long)blockIdx.x - first[i], bp[3 * i].Aimg, bp[3 * i + 1].Aimg, bp[3 * i + 2].Aimg);
}

// nchunk blocks per item: the slices' smallest nodes (bp[3 i].kmin, shared by the orders)
__global__ void __launch_bounds__(256) k_slice_kmin_group(const BesselI8* __restrict__ bp,
                                                        const long* __restrict__ first, int ni) {
  const int i = group_entry(first, ni, blockIdx.x);
  const BesselI8& p = bp[3 * i];
  slice_kmin_body(p.kr, p.K, p.kchunk, (int)(blockIdx.x - first[i]), p.kmin);
}

// ntile_n x (Np / 8) x nchunk blocks per entry (bimg_slice_body)
__global__ void __launch_bounds__(1024) k_bimg_real_group(const BesselI8* __restrict__ bp, const long* __restrict__ first,
                                                       int ne) {
  const int e = group_entry(first, ne, blockIdx.x);
  bimg_slice_body(bp[e], blockIdx.x - first[e]);
}

// ntile_m x ntile_n x nchunk CTAs per entry, radius tile fastest (the CTAs that share a
// column tile's B images run side by side)
__global__ void __launch_bounds__(BI_THREADS, 1) k_gemm_i8_img_group(const BesselI8* __restrict__ bp,
                                                                     const long* __restrict__ first, int ne) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int e = group_entry(first, ne, blockIdx.x);
  const BesselI8& p = bp[e];
  const long b = blockIdx.x - first[e];
  const int mt = (int)(b % p.ntile_m);
  const long rest = b / p.ntile_m;
  gemm_i8_img_body(p, mt, (int)(rest % p.ntile_n), (int)(rest / p.ntile_n), smem);
}

cudaError_t launch_bessel_i8_group(const Synth1DGroup& g, int stage, cudaStream_t s) {
  if (g.ni <= 0) return cudaSuccess;
  const int ne = 3 * g.ni;
  cudaError_t e;
  if (stage == 0 && g.grid[6] > 0) {
    k_slice_kmin_group<<<(unsigned)g.grid[6], 256, 0, s>>>(g.bp, g.first_kmin, g.ni);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (stage == 0 && g.grid[2] > 0) {
    k_aimg_bessel3_group<<<(unsigned)g.grid[2], 256, 0, s>>>(g.bp, g.first_aimg, g.ni);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (stage == 1 && g.grid[3] > 0) {
    k_bimg_real_group<<<(unsigned)g.grid[3], bimg_threads(g.kchunk), 0, s>>>(g.bp, g.first_bimg, ne);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (stage == 2 && g.grid[4] > 0) {
    const size_t sm = bessel_i8_smem(BI_ACC_STRIDE);
    if ((e = cudaFuncSetAttribute(k_gemm_i8_img_group, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) !=
        cudaSuccess)
      return e;
    k_gemm_i8_img_group<<<(unsigned)g.grid[4], BI_THREADS, sm, s>>>(g.bp, g.first_gemm, ne);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ytf

// ytf_mlp_fused.cuh -- the whole forward pass, the whole chain of input gradients and all
// weight gradients of the small MLP, one kernel each, for networks whose layers are at most
// 256 wide (the node placement's 154 -> 256 x 4 -> 2).
//
// k_mlp_chain keeps a 128-row tile of activations (forward) or output gradients (backward) in
// shared memory from the first layer to the last: 128 x 256 values as two BF16 terms (hi, lo) in
// the tensor cores' K-major layout, 128 KB. The BF16 weights come as prepacked images of that
// layout (k_mlp_pack, once per pass), 64 input columns per bulk copy into a 3-slot ring. One
// thread copies and issues the MMAs (hi·W, lo·W per 16 columns, FP32 sums of their own in tensor memory:
// an MMA cuts its sum off at the accumulator's last bit, so the small products would cost a large sum as many
// units as the large ones do. Gradients of 2048 rows 6.0e-6 from 64 bits with one sum, 2.7e-6 with two);
// sixteen warps drain the accumulator, apply bias + GELU (or the GELU derivative), split the result
// and write it over the tile in place. Only the input, the result and what the backward pass
// needs touch global memory.
//   What bounds it: MMAs and drain of a tile alternate (the tile is rewritten in place), about 25
// instructions per value in the drain, and 128 B/clk of shared memory for the operands and the
// weight copies together. 65536 rows of the 154 -> 256 x 4 -> 2 forward pass: 183 us; one launch per
// layer with the operands converted by 128 threads between the MMAs took 2409 us.
//
// k_mlp_dw forms every layer's dW = dZ^T H and db = Σ dZ in one grid over (layer, 128-row tile of
// dW, slice of the batch); k_mlp_dw_sum adds the slices in order. The batch index is the
// contraction index, so a thread takes one column of dZ or H over 8 consecutive samples (coalesced
// loads along the columns) and stores the 8 terms of one K-core as 16 bytes. The bias
// gradient is the sum of the same loads. hi·hi and the two mixed products have sums of their own here too. 8192 rows: 67 us; the GEMMs per layer took 341 us and one
// thread per bias column 961 us.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

#include "ytf_tcgen05.cuh"

namespace ytf {
namespace mlp {

constexpr int FM = 128;         // rows per tile (MMA M)
constexpr int FW = 256;         // widest layer
constexpr int FKB = 64;         // weight columns per ring slot
constexpr int FSLOTS = 3;
constexpr int FMAXL = 16;       // layers
constexpr int FDRAIN = 512;     // drain threads (16 warps) + 1 warp for copies and MMAs
constexpr long FWAIT = 1L << 24;
constexpr uint32_t FPLANE = FM * 64u;  // one 32-column plane of the tile

struct ChainLayer {
  const uint8_t* img;   // packed weights [ceil(K / 64)][2][Np x 64 B]
  int K, N;             // contraction width, outputs
  int ksteps, Np;       // K / 16 and N / 16 rounded up
  const float* bias;    // forward: [N]
  float* Z;             // forward: pre-activations kept for the backward pass (or NULL); backward: read
  float* H;             // forward: activations kept (or NULL); backward: the gradients dZ written
};

struct Chain {
  int L;                // layers run, in order
  int backward;
  long B;
  ChainLayer l[FMAXL];
  const float* X;       // forward: [B][K of the first layer]
  float* out;           // forward: [B][N of the last layer]
  const float* o;       // backward: network outputs [B][2], targets [B][2]
  const float* T;
  float* dout;          // backward: [B][2] output gradient; lb: [B] loss terms
  float* lb;
  unsigned* err;
};

constexpr size_t chain_smem() { return 2ul * 8 * FPLANE + FSLOTS * 2ul * FW * 64 + 128; }

struct ChainShared {
  uint64_t full[FSLOTS], empty[FSLOTS], ready, done;
  uint32_t tmem;
  int stop;
};

__device__ __forceinline__ bool fused_wait(uint32_t bar, uint32_t parity, volatile int* stop, unsigned* err) {
  for (long it = 0; it < FWAIT; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255 && *stop) return false;
  }
  *stop = 1;
  atomicOr(err, 1u);
  return false;
}

// after a wait has given up: lets what the barrier stands for finish (bounded)
__device__ __forceinline__ void fused_drain(uint32_t bar, uint32_t parity) {
  for (long it = 0; it < FWAIT; ++it)
    if (mbar_try(bar, parity)) return;
}

// hi and lo BF16 terms of two values, packed
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - __low2float(h), b - __high2float(h));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred PD;\n\t"
      "setp.ne.b32 PD, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, PD;\n\t}" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

// D F32, A and B BF16, both K-major
__device__ __forceinline__ uint32_t f16_idesc(int Np) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(Np >> 3) << 17) | ((uint32_t)(FM >> 4) << 24);
}

// BF16 weight images: forward rows o, columns i; backward (trans) rows i, columns o. One thread
// per 8 columns of a row (16 bytes of the image), zero outside the matrix.
struct PackLayer {
  const float* W;  // [out][in]
  uint8_t* img;
  int in, out, trans, Np, kblocks;
  long first;      // first thread of this layer
};
struct Pack {
  int n;
  long total;
  PackLayer l[2 * FMAXL];
};
__global__ void __launch_bounds__(256) k_mlp_pack(Pack p) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= p.total) return;
  int e = 0;
  while (e + 1 < p.n && p.l[e + 1].first <= t) ++e;
  const PackLayer& L = p.l[e];
  const int u = (int)(t - L.first);
  const int cores = L.kblocks * (FKB / 8);
  // adjacent threads read adjacent memory: along a row of W, or down a column of it (trans)
  const int row = L.trans ? u % L.Np : u / cores, c = L.trans ? u / L.Np : u % cores;
  const int rows = L.trans ? L.in : L.out, cols = L.trans ? L.out : L.in;
  __nv_bfloat16 v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int k = 8 * c + j;
    const bool in = row < rows && k < cols;
    v[j] = __float2bfloat16_rn(in ? (L.trans ? L.W[(long)k * L.in + row] : L.W[(long)row * L.in + k]) : 0.f);
  }
  uint8_t* dst = L.img + (size_t)(c / 8) * 2 * L.Np * 64 + (size_t)((c / 4) & 1) * L.Np * 64 + plane_off(row, (c & 3) * 16);
  *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
}

// Φ(-t) of t >= 0 (the normal distribution function) without a branch: 2^(t R(t) - 1) with R a
// degree-9 minimax fit of (log2 Φ(-t) + 1) / t on [0, 6] (iteratively reweighted least squares
// against the absolute error of Φ); past t = 6 the exponent keeps falling (-29.9 at 6, to -inf). In FP32 |error| < 7e-8 (rms
// 1.4e-8), as 0.5 (1 + erff) gives, and no cancellation for negative arguments. The library's erff
// branches on its argument, which diverges within a warp and keeps a thread's columns apart: the
// forward pass of 65536 rows took 270 us with it and 186 us with this.
__device__ __forceinline__ float norm_tail(float t) {
  float r = -3.5514208462927854e-08f;
  r = fmaf(r, t, 1.0132938541573822e-06f);
  r = fmaf(r, t, -1.2409629562171176e-05f);
  r = fmaf(r, t, 8.344915113411844e-05f);
  r = fmaf(r, t, -0.0002985420578625053f);
  r = fmaf(r, t, 2.8391224986989982e-05f);
  r = fmaf(r, t, 0.006924435030668974f);
  r = fmaf(r, t, -0.0524333156645298f);
  r = fmaf(r, t, -0.4592214822769165f);
  r = fmaf(r, t, -1.1511043310165405f);
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fmaf(r, t, -1.0f)));
  return e;
}
// z Φ(z) = max(z, 0) - |z| Φ(-|z|)
__device__ __forceinline__ float gelu(float z) { return fmaf(-fabsf(z), norm_tail(fabsf(z)), fmaxf(z, 0.0f)); }
__device__ __forceinline__ float norm_cdf(float z) {
  const float e = norm_tail(fabsf(z));
  return z < 0.0f ? e : 1.0f - e;
}

// columns n .. n + 7 of a row of N values; 16-byte accesses where the rows are aligned (vec)
__device__ __forceinline__ void load_row8(const float* row, int n, int N, bool vec, bool live, float v[8]) {
  if (vec && live && n + 8 <= N) {
    const float4 a = *reinterpret_cast<const float4*>(row + n), c = *reinterpret_cast<const float4*>(row + n + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = live && n + j < N ? row[n + j] : 0.f;
}
__device__ __forceinline__ void store_row8(float* row, int n, int N, bool vec, bool live, const float v[8]) {
  if (!live) return;
  if (vec && n + 8 <= N) {
    *reinterpret_cast<float4*>(row + n) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(row + n + 4) = make_float4(v[4], v[5], v[6], v[7]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (n + j < N) row[n + j] = v[j];
}

template <bool BACK>
__global__ void __launch_bounds__(FDRAIN + 32, 1) k_mlp_chain(const __grid_constant__ Chain p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* hi = smem;
  uint8_t* lo = hi + 8 * FPLANE;
  uint8_t* ring = lo + 8 * FPLANE;
  ChainShared* sh = reinterpret_cast<ChainShared*>(ring + FSLOTS * 2ul * FW * 64);
  volatile int* stop = &sh->stop;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < FSLOTS; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    mbar_init(smem_u32(&sh->ready), FDRAIN / 32);
    mbar_init(smem_u32(&sh->done), 1);
    sh->stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem)),
                 "r"(2 * FW)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;
  const long tiles = (p.B + FM - 1) / FM;

  if (warp == FDRAIN / 32) {
    if (lane == 0) {
      // weight blocks in the order of use, over every tile of this CTA; the copy of block i + 2
      // goes out once block i - 1's MMAs have left its slot
      int per = 0;
      for (int l = 0; l < p.L; ++l) per += (p.l[l].ksteps + 3) / 4;
      const long mine = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
      const long total = mine * per;
      long issued = 0;
      int cl = 0, cb = 0;  // next block to copy
      auto copy_next = [&]() {
        const int slot = (int)(issued % FSLOTS);
        if (issued >= FSLOTS &&
            !fused_wait(smem_u32(&sh->empty[slot]), (uint32_t)((issued / FSLOTS - 1) & 1), stop, p.err))
          return false;
        const ChainLayer& L = p.l[cl];
        const uint32_t bytes = 2u * L.Np * 64u, bar = smem_u32(&sh->full[slot]);
        mbar_arrive_tx(bar, bytes);
        bulk_g2s(smem_u32(ring + (size_t)slot * 2 * FW * 64), L.img + (size_t)cb * bytes, bytes, bar);
        ++issued;
        if (++cb == (L.ksteps + 3) / 4) { cb = 0; cl = cl + 1 == p.L ? 0 : cl + 1; }
        return true;
      };
      bool ok = true;
      while (ok && issued < total && issued < FSLOTS - 1) ok = copy_next();
      long used = 0;
      uint32_t step = 0;  // layers run so far, over all tiles
      for (long t = 0; ok && t < mine; ++t)
        for (int l = 0; ok && l < p.L; ++l, ++step) {
          const ChainLayer& L = p.l[l];
          const uint32_t idesc = f16_idesc(L.Np), planeB = (uint32_t)L.Np * 64u;
          ok = fused_wait(smem_u32(&sh->ready), step & 1, stop, p.err);
          for (int ks = 0; ok && ks < L.ksteps; ks += 4, ++used) {
            const int slot = (int)(used % FSLOTS);
            ok = fused_wait(smem_u32(&sh->full[slot]), (uint32_t)((used / FSLOTS) & 1), stop, p.err);
            if (!ok) break;
            tc_fence_after();
            const uint32_t b0 = smem_u32(ring + (size_t)slot * 2 * FW * 64);
            for (int q = ks; q < min(ks + 4, L.ksteps); ++q) {
              const uint32_t oa = (uint32_t)(q >> 1) * FPLANE + (q & 1) * 256u;
              const uint64_t bd = umma_desc(b0 + (uint32_t)((q >> 1) & 1) * planeB + (q & 1) * 256u);
              mma_f16(tmem, umma_desc(smem_u32(hi) + oa), bd, idesc, q > 0 ? 1u : 0u);
              mma_f16(tmem + FW, umma_desc(smem_u32(lo) + oa), bd, idesc, q > 0 ? 1u : 0u);
            }
            tc_commit(smem_u32(&sh->empty[slot]));
            if (issued < total) ok = copy_next();
          }
          tc_commit(smem_u32(&sh->done));
        }
      // every issued copy lands and every issued MMA ends before the CTA exits
      for (long s = issued > FSLOTS ? issued - FSLOTS : 0; s < issued; ++s)
        fused_drain(smem_u32(&sh->full[s % FSLOTS]), (uint32_t)((s / FSLOTS) & 1));
      // `step` layers were committed to `done` (a broken one too)
      if (!ok && step > 0) fused_drain(smem_u32(&sh->done), (step - 1) & 1);
    }
  } else {
    const int q4 = warp & 3, part = warp >> 2;
    const uint32_t lanebase = (uint32_t)(32 * q4) << 16;
    uint32_t step = 0;
    bool ok = true;
    for (long tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
      const long row0 = tile * FM;
      // the tile's first operand
      if (BACK) {
        if (part == 0) {  // loss terms and the output gradient of one sample per thread
          const int r = 32 * q4 + lane;
          const long b = row0 + r;
          float g0 = 0.f, g1 = 0.f;
          if (b < p.B) {
            const float o0 = p.o[2 * b], o1 = p.o[2 * b + 1], t0 = p.T[2 * b], t1 = p.T[2 * b + 1];
            const float e = o0 - t0;
            const float sp = o1 > 0 ? o1 + log1pf(expf(-o1)) : log1pf(expf(o1));
            p.lb[b] = e * e + (sp - t1 * o1);
            const float sig = 1.f / (1.f + expf(-o1));
            const int n = (int)p.B;
            g0 = 2.f * e / n;
            g1 = (sig - t1) / n;
            p.dout[2 * b] = g0;
            p.dout[2 * b + 1] = g1;
          }
          uint32_t h, w;
          split2(g0, g1, h, w);
          const uint4 z = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(hi + plane_off(r, 0)) = make_uint4(h, 0, 0, 0);
          *reinterpret_cast<uint4*>(lo + plane_off(r, 0)) = make_uint4(w, 0, 0, 0);
          *reinterpret_cast<uint4*>(hi + plane_off(r, 16)) = z;
          *reinterpret_cast<uint4*>(lo + plane_off(r, 16)) = z;
        }
      } else {
        const int K = p.l[0].K, groups = p.l[0].ksteps * 2;  // 8-column groups
        const int rr = lane >> 2, kk = 2 * (lane & 3);
        // a warp takes 8 rows x 8 columns: 32-byte runs of the rows, 128-byte runs of a plane;
        // 8 such units are loaded before any is converted (one by one the DRAM latencies add up)
        for (int u0 = warp; u0 < 16 * groups; u0 += 8 * (FDRAIN / 32)) {
          float v0[8], v1[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int u = u0 + i * (FDRAIN / 32), r = 8 * (u & 15) + rr, k = 8 * (u >> 4) + kk;
            const long b = row0 + r;
            const float* x = p.X + b * K + k;
            v0[i] = b < p.B && k < K ? __ldg(x) : 0.f;
            v1[i] = b < p.B && k + 1 < K ? __ldg(x + 1) : 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int u = u0 + i * (FDRAIN / 32), r = 8 * (u & 15) + rr, k = 8 * (u >> 4) + kk;
            if (u >= 16 * groups) break;
            uint32_t h, w;
            split2(v0[i], v1[i], h, w);
            const uint32_t off = (uint32_t)(k >> 5) * FPLANE + plane_off(r, 2 * (k & 31));
            *reinterpret_cast<uint32_t*>(hi + off) = h;
            *reinterpret_cast<uint32_t*>(lo + off) = w;
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->ready));
      for (int l = 0; l < p.L; ++l, ++step) {
        const ChainLayer& L = p.l[l];
        ok = fused_wait(smem_u32(&sh->done), step & 1, stop, p.err);
        ok = __all_sync(0xffffffffu, ok && !*stop);
        if (!ok) break;
        tc_fence_after();
        const int r = 32 * q4 + lane;
        const long b = row0 + r;
        const bool live = b < p.B;
        const bool last = l + 1 == p.L;
        const bool vec = (L.N & 3) == 0;  // rows of Z and H start on 16 bytes
        const bool bvec = (reinterpret_cast<uintptr_t>(L.bias) & 15) == 0;
        // two 8-column groups at a time (independent chains hide the latencies)
        constexpr int NG = FDRAIN / 128;
        for (int n0 = 8 * part; n0 < L.Np; n0 += 16 * NG) {
          const bool two = n0 + 8 * NG < L.Np;
          uint32_t v[2][8], w[2][8];
          tmem_ld8(tmem + lanebase + n0, v[0]);
          tmem_ld8(tmem + FW + lanebase + n0, w[0]);
          if (two) {
            tmem_ld8(tmem + lanebase + n0 + 8 * NG, v[1]);
            tmem_ld8(tmem + FW + lanebase + n0 + 8 * NG, w[1]);
          }
          float z[2][8], y[2][8];  // BACK: Z; forward: the bias, then Z
          const float* zrow = BACK ? L.Z + b * L.N : L.bias;
          load_row8(zrow, n0, L.N, BACK ? vec : bvec, BACK ? live : true, z[0]);
          if (two) load_row8(zrow, n0 + 8 * NG, L.N, BACK ? vec : bvec, BACK ? live : true, z[1]);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (g == 1 && !two) break;
            const int n = n0 + 8 * NG * g;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float acc = __uint_as_float(v[g][j]) + __uint_as_float(w[g][j]);
              if (BACK) {
                // dZ = dH GELU'(Z), GELU'(z) = Φ(z) + z φ(z)
                const float zz = z[g][j];
                y[g][j] = acc * fmaf(zz * 0.39894228040143268f, expf(-0.5f * zz * zz), norm_cdf(zz));
              } else {
                z[g][j] += acc;
                y[g][j] = last ? z[g][j] : gelu(z[g][j]);
              }
            }
            if (n + 8 > L.N)  // past the layer's width the next operand is zero
#pragma unroll
              for (int j = 0; j < 8; ++j) y[g][j] = n + j < L.N ? y[g][j] : 0.f;
            if (!BACK && L.Z) store_row8(L.Z + b * L.N, n, L.N, vec, live, z[g]);
            if (L.H) store_row8(L.H + b * L.N, n, L.N, vec, live, y[g]);
            if (!BACK && last) store_row8(p.out + b * L.N, n, L.N, false, live, y[g]);
            if (!last) {
              uint4 h, l4;
              split2(y[g][0], y[g][1], h.x, l4.x);
              split2(y[g][2], y[g][3], h.y, l4.y);
              split2(y[g][4], y[g][5], h.z, l4.z);
              split2(y[g][6], y[g][7], h.w, l4.w);
              const uint32_t off = (uint32_t)(n >> 5) * FPLANE + plane_off(r, 2 * (n & 31));
              *reinterpret_cast<uint4*>(hi + off) = h;
              *reinterpret_cast<uint4*>(lo + off) = l4;
            }
          }
        }
        // the accumulator is read and the next operand written before the next MMAs
        tc_fence_before();
        if (!last) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh->ready));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * FW) : "memory");
  }
}

// ------------------------------------------------------------------------------------
// weight and bias gradients
// ------------------------------------------------------------------------------------
struct DwLayer {
  const float *dZ, *H;  // [B][M], [B][N]
  int M, N, Np;         // out, in, in rounded up to 16
  int mtiles;
  int first;            // first block of this layer (blocks: mtiles x slices, tile fastest)
  long poff;            // offset of its weights in a slice's parameter block
  long boff;            // and of its biases
};
struct Dw {
  int L, slices, blocks;
  long B, slice;        // batch rows per slice (a multiple of 64)
  long nparam;
  float* part;          // [slices][nparam]
  float* g;             // [nparam]
  unsigned* err;
  DwLayer l[FMAXL];
};
constexpr int DW_THREADS = 512;
constexpr uint32_t DW_STAGE = 2u * (2u * FPLANE + 2u * FW * 64u);  // 64 samples: A and B, hi and lo
constexpr size_t dw_smem() { return 2ul * DW_STAGE + 4ul * DW_THREADS + 64; }

// 8 consecutive samples of one column; as the 16 bytes of a K-core in the hi and lo planes
__device__ __forceinline__ void dw_load(const float* src, long ld, long b0, long b1, bool live, float v[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = live && b0 + j < b1 ? __ldg(src + (b0 + j) * ld) : 0.f;
}
__device__ __forceinline__ void dw_store(const float v[8], uint8_t* hi, uint8_t* lo, uint32_t off) {
  uint4 h, w;
  split2(v[0], v[1], h.x, w.x);
  split2(v[2], v[3], h.y, w.y);
  split2(v[4], v[5], h.z, w.z);
  split2(v[6], v[7], h.w, w.w);
  *reinterpret_cast<uint4*>(hi + off) = h;
  *reinterpret_cast<uint4*>(lo + off) = w;
}

__global__ void __launch_bounds__(DW_THREADS, 1) k_mlp_dw(const __grid_constant__ Dw p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_sh;
  __shared__ int stop_sh;
  volatile int* stop = &stop_sh;
  float* dbs = reinterpret_cast<float*>(smem + 2ul * DW_STAGE);  // [4][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int e = 0;
  while (e + 1 < p.L && p.l[e + 1].first <= (int)blockIdx.x) ++e;
  const DwLayer& L = p.l[e];
  const int u = (int)blockIdx.x - L.first, mt = u % L.mtiles, sl = u / L.mtiles;
  const long s0 = (long)sl * p.slice, s1 = min(p.B, s0 + p.slice);
  const int nkb = s1 > s0 ? (int)((s1 - s0 + 63) / 64) : 0;
  if (tid == 0) {
    mbar_init(smem_u32(&bar[0]), 1);
    mbar_init(smem_u32(&bar[1]), 1);
    stop_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(2 * FW)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_sh, planeB = (uint32_t)L.Np * 64u, idesc = f16_idesc(L.Np);
  // this thread's columns and K-cores (8 samples) of a 64-sample block: dZ column ma, cores
  // tid >> 7 and + 4; H column nb, cores tid >> 8 and + 2, + 4, + 6
  const int ma = tid & 127, nb = tid & 255;
  const bool alive = mt * FM + ma < L.M, blive = nb < L.N;
  float db = 0.f;
  bool ok = true;
  int kb = 0;
  for (; kb < nkb; ++kb) {
    uint8_t* st = smem + (kb & 1) * DW_STAGE;
    uint8_t *ah = st, *al = ah + 2 * FPLANE, *bh = al + 2 * FPLANE, *bl = bh + 2 * planeB;
    const long b0 = s0 + 64L * kb;
    float va[2][8], vb[4][8];
#pragma unroll
    for (int i = 0; i < 2; ++i) dw_load(L.dZ + mt * FM + ma, L.M, b0 + 8 * ((tid >> 7) + 4 * i), s1, alive, va[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) dw_load(L.H + nb, L.N, b0 + 8 * ((tid >> 8) + 2 * i), s1, blive, vb[i]);
    // the MMAs that read this buffer two blocks ago are done
    if (kb >= 2) ok = fused_wait(smem_u32(&bar[kb & 1]), (uint32_t)((kb >> 1) - 1) & 1, stop, p.err);
    if (!__syncthreads_and(ok)) { ok = false; break; }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) db += va[i][j];
      const int core = (tid >> 7) + 4 * i;
      dw_store(va[i], ah, al, (uint32_t)(core >> 2) * FPLANE + plane_off(ma, 16 * (core & 3)));
    }
    if (nb < L.Np)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int core = (tid >> 8) + 2 * i;
        dw_store(vb[i], bh, bl, (uint32_t)(core >> 2) * planeB + plane_off(nb, 16 * (core & 3)));
      }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t oa = (uint32_t)(q >> 1) * FPLANE + (q & 1) * 256u, ob = (uint32_t)(q >> 1) * planeB + (q & 1) * 256u;
        const uint64_t dah = umma_desc(smem_u32(ah) + oa), dal = umma_desc(smem_u32(al) + oa);
        const uint64_t dbh = umma_desc(smem_u32(bh) + ob), dbl = umma_desc(smem_u32(bl) + ob);
        mma_f16(tmem, dah, dbh, idesc, kb > 0 || q > 0 ? 1u : 0u);
        mma_f16(tmem + FW, dah, dbl, idesc, kb > 0 || q > 0 ? 1u : 0u);
        mma_f16(tmem + FW, dal, dbh, idesc, 1u);
      }
      tc_commit(smem_u32(&bar[kb & 1]));
    }
  }
  // the last block's commit covers every earlier MMA
  if (kb > 0) {
    if (ok) ok = fused_wait(smem_u32(&bar[(kb - 1) & 1]), (uint32_t)((kb - 1) >> 1) & 1, stop, p.err);
    else fused_drain(smem_u32(&bar[(kb - 1) & 1]), (uint32_t)((kb - 1) >> 1) & 1);
  }
  ok = __syncthreads_and(ok);
  tc_fence_after();
  float* part = p.part + (long)sl * p.nparam;
  if (ok) {
    const int q4 = warp & 3;
    const int m = mt * FM + 32 * q4 + lane;
    for (int n = 8 * (warp >> 2); n < L.Np; n += 8 * (DW_THREADS / 128)) {
      uint32_t v[8], w[8];
      if (nkb > 0) {
        tmem_ld8(tmem + ((uint32_t)(32 * q4) << 16) + n, v);
        tmem_ld8(tmem + FW + ((uint32_t)(32 * q4) << 16) + n, w);
        tmem_wait_ld();
      }
      if (m < L.M)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (n + j < L.N) part[L.poff + (long)m * L.N + n + j] = nkb > 0 ? __uint_as_float(v[j]) + __uint_as_float(w[j]) : 0.f;
    }
  }
  dbs[tid] = db;
  __syncthreads();
  if (tid < 128 && alive) part[L.boff + mt * FM + tid] = (dbs[tid] + dbs[128 + tid]) + (dbs[256 + tid] + dbs[384 + tid]);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * FW) : "memory");
  }
}

__global__ void __launch_bounds__(256) k_mlp_dw_sum(long n, int slices, const float* __restrict__ part,
                                                    float* __restrict__ g) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  float s = 0.f;
  for (int i = 0; i < slices; ++i) s += part[(long)i * n + t];
  g[t] = s;
}

}  // namespace mlp
}  // namespace ytf

// ytf_mlp.cu -- the small MLP of the learned node placement: forward, backward and Adam
// kernels, and its C ABI.
//
// Network: L linear layers (sizes n_0 -> n_1 -> ... -> n_L), GELU after every layer but the
// last. Master parameters are FP32 (W_l [n_l x n_{l-1}] row-major, then b_l [n_l], layer by
// layer); every forward/backward pass first rounds the weights to BF16 and multiplies with
// those, accumulating in FP32 ("BF16 weights, FP32 accumulation"). Activations and gradients
// are FP32. Loss over a batch of B samples with targets (t0, t1):
//   ℓ = mean_b (o0 - t0)^2 + mean_b [softplus(o1) - t1 o1]
// (o0: the log-response prediction, o1: the logit of the pole-proximity score).
//
// Networks whose layers are at most 256 wide run fused (ytf_mlp_fused.cuh): one kernel for the
// forward pass, one for the input gradients, one for all weight gradients. Wider ones take one
// strided GEMM per product of a layer:
//   forward  Z[b][o]  = Σ_i H[b][i] W[o][i] + bias[o]   (then GELU)
//   input    dH[b][i] = Σ_o dZ[b][o] W[o][i]
//   weights  dW[o][i] = Σ_b dZ[b][o] H[b][i]
// C[m][n] = Σ_k A(m, k) B(k, n), A(m, k) = A[m sam + k sak], B(k, n) = B[k sbk + n sbn], on the
// tensor cores (tcgen05.mma kind::f16, BF16 operands, FP32 accumulation in tensor memory). The
// BF16 weights enter as they are; an FP32 operand (activations, gradients) is split into two
// BF16 terms hi = bf16(v), lo = bf16(v - hi), and the products hi·hi, hi·lo, lo·hi are summed,
// so an FP32 operand keeps about 16 significant bits (the dropped lo·lo is below 2^-16 of it).
// A CTA computes a 128 x Np tile (Np = N rounded up to 16, at most 256) over K in blocks of
// 128: its 128 threads convert the block's operands into shared memory (planes of 64-byte rows,
// 32 BF16 each, the canonical no-swizzle K-major layout), one thread issues the block's MMAs,
// their commit frees the buffers for the next block; the 4 warps then drain the accumulator
// (warp w: tensor-memory lanes 32w..32w+31 = the tile's rows) with bias, accumulation and GELU.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/ytf.h"
#include "ytf_mlp_fused.cuh"
#include "ytf_tcgen05.cuh"

namespace ytf {
namespace mlp {

constexpr int GM = 128;          // tile rows (MMA M)
constexpr int GNMAX = 256;       // largest tile width (MMA N)
constexpr int GKB = 128;         // K per block: 4 planes of 32
constexpr long GWAIT = 1L << 24; // polls of the bounded commit wait

__device__ __forceinline__ uint32_t plane_bf(int r, int k) { return plane_off(r, 2 * k); }

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred PD;\n\t"
      "setp.ne.b32 PD, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, PD;\n\t}" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

// the two BF16 terms of a source value (the second is 0 for a BF16 source)
__device__ __forceinline__ void split_bf(float v, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(v);
  lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// tn: the tile width (128 or 256). With ksl > 0 the K range is split: CTA (x, y, z) sums
// K in [z ksl, (z + 1) ksl) and writes its raw sums to part[z][M][N] (k_splitk_finish adds
// the slices, the bias, the accumulation and GELU); otherwise it finishes the tile itself.
template <class TA, class TB>
__global__ void __launch_bounds__(128, 1) k_gemm_tc(int M, int N, int K, const TA* __restrict__ A, long sam, long sak,
                                                     const TB* __restrict__ B, long sbk, long sbn,
                                                     float* __restrict__ C, long ldc, const float* __restrict__ bias,
                                                     float* __restrict__ H, int act, int accumulate, int tn, int ksl,
                                                     float* __restrict__ part, unsigned* __restrict__ err) {
  constexpr bool SA = std::is_same<TA, float>::value;  // split A into two terms
  constexpr bool SB = std::is_same<TB, float>::value;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t done;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * GM, n0 = blockIdx.x * tn;
  const int nt = min(tn, N - n0);
  const int kbeg = ksl > 0 ? (int)blockIdx.z * ksl : 0;
  const int kend = ksl > 0 ? min(K, kbeg + ksl) : K;
  const int Np = ((nt + 15) / 16) * 16;
  const uint32_t planeA = GM * 64u, planeB = (uint32_t)Np * 64u;
  constexpr int NPL = GKB / 32;
  uint8_t* Ahi = smem;
  uint8_t* Alo = Ahi + NPL * planeA;
  uint8_t* Bhi = Alo + (SA ? NPL * planeA : 0);
  uint8_t* Blo = Bhi + NPL * planeB;
  if (tid == 0) {
    mbar_init(smem_u32(&done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(GNMAX)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  // kind::f16: D F32 (bit 4), A BF16 (bits 7-9 = 1), B BF16 (bits 10-12 = 1), both K-major
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(Np >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
  bool ok = true;
  int round = 0;
  for (int k0 = kbeg; k0 < kend; k0 += GKB, ++round) {
    if (round > 0) {
      // the previous block's MMAs have read the buffers before they are overwritten
      bool got = false;
      for (long it = 0; it < GWAIT && !got; ++it) got = mbar_try(smem_u32(&done), (round - 1) & 1);
      if (!got) { ok = false; if (tid == 0) atomicOr(err, 1u); break; }
    }
    for (int e = tid; e < GM * GKB; e += 128) {
      int r, k;
      if (sak == 1) { r = e / GKB; k = e % GKB; } else { k = e / GM; r = e % GM; }
      const int m = m0 + r, kk = k0 + k;
      const float v = (m < M && kk < kend) ? (float)A[(long)m * sam + (long)kk * sak] : 0.f;
      __nv_bfloat16 hi, lo;
      split_bf(v, hi, lo);
      const uint32_t off = (k >> 5) * planeA + plane_bf(r, k & 31);
      *reinterpret_cast<__nv_bfloat16*>(Ahi + off) = hi;
      if (SA) *reinterpret_cast<__nv_bfloat16*>(Alo + off) = lo;
    }
    for (int e = tid; e < Np * GKB; e += 128) {
      int r, k;
      if (sbk == 1) { r = e / GKB; k = e % GKB; } else { k = e / Np; r = e % Np; }
      const int n = n0 + r, kk = k0 + k;
      const float v = (r < nt && kk < kend) ? (float)B[(long)kk * sbk + (long)n * sbn] : 0.f;
      __nv_bfloat16 hi, lo;
      split_bf(v, hi, lo);
      const uint32_t off = (k >> 5) * planeB + plane_bf(r, k & 31);
      *reinterpret_cast<__nv_bfloat16*>(Bhi + off) = hi;
      if (SB) *reinterpret_cast<__nv_bfloat16*>(Blo + off) = lo;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int pl = 0; pl < NPL; ++pl)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t oa = pl * planeA + t * 256u, ob = pl * planeB + t * 256u;
          // the first MMA of the tile overwrites the accumulator, every other one adds to it
          mma_bf16(tmem, umma_desc(smem_u32(Ahi + oa)), umma_desc(smem_u32(Bhi + ob)), idesc,
                   (k0 > kbeg || pl > 0 || t > 0) ? 1u : 0u);
          if (SB) mma_bf16(tmem, umma_desc(smem_u32(Ahi + oa)), umma_desc(smem_u32(Blo + ob)), idesc, 1u);
          if (SA) mma_bf16(tmem, umma_desc(smem_u32(Alo + oa)), umma_desc(smem_u32(Bhi + ob)), idesc, 1u);
        }
      tc_commit(smem_u32(&done));
    }
  }
  // the last block's MMAs (and with them every earlier one) complete before the drain
  if (round > 0) {
    bool got = false;
    for (long it = 0; it < GWAIT && !got; ++it) got = mbar_try(smem_u32(&done), (round - 1) & 1);
    if (!got) { ok = false; if (tid == 0) atomicOr(err, 1u); }
  }
  ok = __all_sync(0xffffffffu, ok);
  tc_fence_after();
  if (ok && round > 0) {
    const int m = m0 + 32 * warp + lane;
    const uint32_t lanebase = (uint32_t)(32 * warp) << 16;
    for (int c0 = 0; c0 < Np; c0 += 8) {
      uint32_t v[8];
      tmem_ld8(tmem + lanebase + c0, v);
      tmem_wait_ld();
      if (m < M) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int n = n0 + c0 + j;
          if (c0 + j >= nt) break;
          if (part) {
            part[((long)blockIdx.z * M + m) * N + n] = __uint_as_float(v[j]);
            continue;
          }
          float z = __uint_as_float(v[j]) + (bias ? bias[n] : 0.f);
          if (accumulate) z += C[(long)m * ldc + n];
          C[(long)m * ldc + n] = z;
          if (H) H[(long)m * ldc + n] = act ? 0.5f * z * (1.f + erff(z * 0.70710678118654752f)) : z;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GNMAX) : "memory");
}

// the K slices of a split GEMM summed in slice order, then bias, accumulation and GELU
__global__ void k_splitk_finish(int M, int N, int S, const float* __restrict__ part, float* __restrict__ C, long ldc,
                                const float* __restrict__ bias, float* __restrict__ H, int act, int accumulate) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)M * N) return;
  const int m = (int)(t / N), n = (int)(t % N);
  float z = 0.f;
  for (int sl = 0; sl < S; ++sl) z += part[(long)sl * M * N + t];
  z += bias ? bias[n] : 0.f;
  if (accumulate) z += C[(long)m * ldc + n];
  C[(long)m * ldc + n] = z;
  if (H) H[(long)m * ldc + n] = act ? 0.5f * z * (1.f + erff(z * 0.70710678118654752f)) : z;
}

template <class TA, class TB>
size_t gemm_tc_smem(int Np) {
  constexpr bool SA = std::is_same<TA, float>::value, SB = std::is_same<TB, float>::value;
  return (size_t)(GKB / 32) * ((SA ? 2 : 1) * GM * 64 + (SB ? 2 : 1) * (size_t)Np * 64);
}

// dZ = dH * GELU'(Z), GELU'(z) = Φ(z) + z φ(z)
__global__ void k_gelu_back(long n, const float* __restrict__ Z, const float* __restrict__ dH, float* __restrict__ dZ) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float z = Z[t];
  const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  dZ[t] = dH[t] * (cdf + z * pdf);
}

// column sums: db[o] = Σ_b dZ[b][o]
__global__ void k_colsum(int B, int N, const float* __restrict__ dZ, float* __restrict__ db) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= N) return;
  float s = 0.f;
  for (int b = 0; b < B; ++b) s += dZ[(long)b * N + o];
  db[o] = s;
}

// loss terms and the output gradient; out: [B][2], T: [B][2]; per-sample loss into lb
__global__ void k_loss(int B, const float* __restrict__ out, const float* __restrict__ T, float* __restrict__ dout,
                       float* __restrict__ lb) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const float o0 = out[2 * b], o1 = out[2 * b + 1], t0 = T[2 * b], t1 = T[2 * b + 1];
  const float e = o0 - t0;
  const float sp = o1 > 0 ? o1 + log1pf(expf(-o1)) : log1pf(expf(o1));
  lb[b] = e * e + (sp - t1 * o1);
  const float sig = 1.f / (1.f + expf(-o1));
  dout[2 * b] = 2.f * e / B;
  dout[2 * b + 1] = (sig - t1) / B;
}

// a mini-batch drawn with replacement from the device-resident set: sample index from a
// counter-based hash (splitmix64) of (seed, step, row)
__global__ void k_gather(int B, int d, long n, unsigned long long seed, long step, const float* __restrict__ X,
                         const float* __restrict__ T, float* __restrict__ Xb, float* __restrict__ Tb) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)B * (d + 2)) return;
  const int b = (int)(t / (d + 2)), c = (int)(t % (d + 2));
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(step * B + b + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  const long i = (long)(z % (unsigned long long)n);
  if (c < d) Xb[(long)b * d + c] = X[i * d + c];
  else Tb[2L * b + (c - d)] = T[2 * i + (c - d)];
}

__global__ void k_to_bf16(long n, const float* __restrict__ a, __nv_bfloat16* __restrict__ b) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) b[t] = __float2bfloat16_rn(a[t]);
}

__global__ void k_adam(long n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float gt = g[t];
  const float mt = b1 * m[t] + (1.f - b1) * gt;
  const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
  m[t] = mt;
  v[t] = vt;
  p[t] -= lr * (mt / c1) / (sqrtf(vt / c2) + eps);
}

}  // namespace mlp
}  // namespace ytf

using namespace ytf::mlp;

struct ytf_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::vector<int> sizes;          // n_0 .. n_L
  std::vector<long> woff, boff;    // offsets of W_l and b_l in the parameter vector
  long nparam = 0;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16* wb = nullptr;     // BF16 copy of the parameters (weights used from here)
  long step = 0;
  // activations for the largest batch seen: Z_l and H_l per layer, gradients, loss terms
  long cap = 0;
  std::vector<float*> Z, H, dZ, dH;
  float *T = nullptr, *lb = nullptr;
  // inputs and outputs of the largest forward-only batch that is copied (fused networks)
  long cap_io = 0;
  float *Xin = nullptr, *Yout = nullptr;
  unsigned* tc_err = nullptr;      // page-locked: set by a kernel whose tensor-core wait ran out
  float* part = nullptr;           // K-slice sums of split GEMMs, batch-slice sums of the gradients
  size_t part_cap = 0;
  bool fused = false;              // every layer at most 256 wide (ytf_mlp_fused.cuh)
  uint8_t* img = nullptr;          // packed BF16 weights: forward images, then transposed ones
  std::vector<size_t> img_f, img_b;
  int nsm = 148;
  std::string err;
  ~ytf_mlp() {
    cudaFree(p); cudaFree(g); cudaFree(m); cudaFree(v); cudaFree(wb);
    for (auto* q : Z) cudaFree(q);
    for (auto* q : H) cudaFree(q);
    for (auto* q : dZ) cudaFree(q);
    for (auto* q : dH) cudaFree(q);
    cudaFree(T); cudaFree(lb); cudaFree(Xin); cudaFree(Yout); cudaFree(part); cudaFree(img);
    if (tc_err) cudaFreeHost(tc_err);
  }
};

namespace {

int mfail(ytf_mlp* n, int code, const std::string& msg) {
  if (n) n->err = msg;
  return code;
}
#define MCK(call)                                                                    \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) return mfail(net, YTF_ERR_CUDA, cudaGetErrorString(e_)); \
  } while (0)

template <class TA, class TB>
cudaError_t gemm(ytf_mlp* net, int M, int N, int K, const TA* A, long sam, long sak, const TB* B, long sbk, long sbn,
                 float* C, long ldc, const float* bias, float* H, int act, int accumulate) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  // fill the 148 SMs: 128-wide tiles when 256-wide ones are too few, then K slices
  const int mt = (M + GM - 1) / GM;
  const int tn = (long)mt * ((N + GNMAX - 1) / GNMAX) < 148 && N > 128 ? 128 : GNMAX;
  const int tiles = mt * ((N + tn - 1) / tn);
  int S = 1, ksl = 0;
  if (tiles < 74 && K >= 2 * GKB) {
    S = std::min((148 + tiles - 1) / tiles, (K + GKB - 1) / GKB);
    ksl = (((K + S - 1) / S + GKB - 1) / GKB) * GKB;
    S = (K + ksl - 1) / ksl;
  }
  float* part = nullptr;
  if (S > 1) {
    const size_t need = (size_t)S * M * N;
    if (need > net->part_cap) {
      cudaFree(net->part);
      net->part = nullptr;
      net->part_cap = 0;
      cudaError_t e = cudaMalloc(&net->part, sizeof(float) * need);
      if (e != cudaSuccess) return e;
      net->part_cap = need;
    }
    part = net->part;
  } else {
    ksl = 0;
  }
  const int Np = ((std::min(N, tn) + 15) / 16) * 16;
  const size_t sm = gemm_tc_smem<TA, TB>(Np);
  cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  dim3 grid((N + tn - 1) / tn, mt, S);
  k_gemm_tc<TA, TB><<<grid, 128, sm, net->stream>>>(M, N, K, A, sam, sak, B, sbk, sbn, C, ldc, bias, H, act, accumulate,
                                                   tn, ksl, part, net->tc_err);
  if ((e = cudaGetLastError()) != cudaSuccess || S == 1) return e;
  k_splitk_finish<<<(unsigned)(((long)M * N + 255) / 256), 256, 0, net->stream>>>(M, N, S, part, C, ldc, bias, H, act,
                                                                              accumulate);
  return cudaGetLastError();
}

int ensure(ytf_mlp* net, long B) {
  if (B <= net->cap) return YTF_OK;
  for (auto* q : net->Z) cudaFree(q);
  for (auto* q : net->H) cudaFree(q);
  for (auto* q : net->dZ) cudaFree(q);
  for (auto* q : net->dH) cudaFree(q);
  cudaFree(net->T); cudaFree(net->lb);
  net->T = net->lb = nullptr;
  net->cap = 0;
  const int L = (int)net->sizes.size() - 1;
  net->Z.assign(L + 1, nullptr); net->H.assign(L + 1, nullptr);
  net->dZ.assign(L + 1, nullptr); net->dH.assign(L + 1, nullptr);
  for (int l = 0; l <= L; ++l) {
    const size_t bytes = sizeof(float) * B * net->sizes[l];
    MCK(cudaMalloc(&net->H[l], bytes));
    if (!net->fused) MCK(cudaMalloc(&net->dH[l], bytes));
    if (l > 0) {
      MCK(cudaMalloc(&net->Z[l], bytes));
      MCK(cudaMalloc(&net->dZ[l], bytes));
    }
  }
  MCK(cudaMalloc(&net->T, sizeof(float) * 2 * B));
  MCK(cudaMalloc(&net->lb, sizeof(float) * B));
  net->cap = B;
  return YTF_OK;
}

// staging of a forward-only batch from host memory or with outputs over its inputs
int ensure_io(ytf_mlp* net, long B) {
  if (B <= net->cap_io) return YTF_OK;
  cudaFree(net->Xin); cudaFree(net->Yout);
  net->Xin = net->Yout = nullptr;
  net->cap_io = 0;
  MCK(cudaMalloc(&net->Xin, sizeof(float) * B * net->sizes[0]));
  MCK(cudaMalloc(&net->Yout, sizeof(float) * B * net->sizes.back()));
  net->cap_io = B;
  return YTF_OK;
}

// memory of another GPU, which a kernel of this one reaches only with peer access (a copy always does)
bool other_device(int device, const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice && a.device != device;
}

int round16(int n) { return (n + 15) / 16 * 16; }

// the weight images of the fused kernels from the current parameters
int pack_weights(ytf_mlp* net, bool back) {
  const int L = (int)net->sizes.size() - 1;
  Pack pk;
  pk.n = 0;
  pk.total = 0;
  for (int trans = 0; trans <= (back ? 1 : 0); ++trans)
    for (int l = 1 + trans; l <= L; ++l) {  // the first layer's input gradient is not formed
      PackLayer& q = pk.l[pk.n++];
      q.W = net->p + net->woff[l - 1];
      q.img = net->img + (trans ? net->img_b[l - 1] : net->img_f[l - 1]);
      q.in = net->sizes[l - 1];
      q.out = net->sizes[l];
      q.trans = trans;
      q.Np = round16(trans ? q.in : q.out);
      q.kblocks = ((trans ? q.out : q.in) + FKB - 1) / FKB;
      q.first = pk.total;
      pk.total += (long)q.Np * q.kblocks * (FKB / 8);
    }
  k_mlp_pack<<<(unsigned)((pk.total + 255) / 256), 256, 0, net->stream>>>(pk);
  MCK(cudaGetLastError());
  return YTF_OK;
}

// forward pass of B device rows X into `out`; `keep`: Z_l and H_l of the inner layers for the backward pass
int forward_fused(ytf_mlp* net, long B, const float* X, float* out, bool keep) {
  const int L = (int)net->sizes.size() - 1;
  Chain c;
  std::memset(&c, 0, sizeof(c));
  c.L = L;
  c.B = B;
  c.X = X;
  c.out = out;
  c.err = net->tc_err;
  for (int l = 1; l <= L; ++l) {
    ChainLayer& q = c.l[l - 1];
    q.img = net->img + net->img_f[l - 1];
    q.K = net->sizes[l - 1];
    q.N = net->sizes[l];
    q.ksteps = round16(q.K) / 16;
    q.Np = round16(q.N);
    q.bias = net->p + net->boff[l - 1];
    if (keep && l < L) { q.Z = net->Z[l]; q.H = net->H[l]; }
  }
  MCK(cudaFuncSetAttribute(k_mlp_chain<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem()));
  const long tiles = (B + FM - 1) / FM;
  k_mlp_chain<false><<<(unsigned)std::min<long>(tiles, net->nsm), FDRAIN + 32, chain_smem(), net->stream>>>(c);
  MCK(cudaGetLastError());
  return YTF_OK;
}

// gradients into g from the inputs in X, the kept activations, the outputs in H[L] and the targets in T
int backward_fused(ytf_mlp* net, long B, const float* X) {
  const int L = (int)net->sizes.size() - 1;
  Chain c;
  std::memset(&c, 0, sizeof(c));
  c.L = L - 1;
  c.backward = 1;
  c.B = B;
  c.o = net->H[L];
  c.T = net->T;
  c.dout = net->dZ[L];
  c.lb = net->lb;
  c.err = net->tc_err;
  for (int l = L; l >= 2; --l) {  // dZ_{l-1} = (dZ_l W_l) GELU'(Z_{l-1})
    ChainLayer& q = c.l[L - l];
    q.img = net->img + net->img_b[l - 1];
    q.K = net->sizes[l];
    q.N = net->sizes[l - 1];
    q.ksteps = round16(q.K) / 16;
    q.Np = round16(q.N);
    q.Z = net->Z[l - 1];
    q.H = net->dZ[l - 1];
  }
  MCK(cudaFuncSetAttribute(k_mlp_chain<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem()));
  const long tiles = (B + FM - 1) / FM;
  k_mlp_chain<true><<<(unsigned)std::min<long>(tiles, net->nsm), FDRAIN + 32, chain_smem(), net->stream>>>(c);
  MCK(cudaGetLastError());
  Dw d;
  std::memset(&d, 0, sizeof(d));
  d.L = L;
  d.B = B;
  d.nparam = net->nparam;
  d.g = net->g;
  d.err = net->tc_err;
  int mtiles = 0;
  for (int l = 1; l <= L; ++l) mtiles += (net->sizes[l] + FM - 1) / FM;
  // batch slices of at least 64 samples that fill the SMs once (one CTA per SM: 192 KB of operands)
  const long want = std::max(1, net->nsm / mtiles);
  d.slice = std::max(64L, ((B + want - 1) / want + 63) / 64 * 64);
  d.slices = (int)((B + d.slice - 1) / d.slice);
  const size_t need = (size_t)d.slices * net->nparam;
  if (need > net->part_cap) {
    cudaFree(net->part);
    net->part = nullptr;
    net->part_cap = 0;
    MCK(cudaMalloc(&net->part, sizeof(float) * need));
    net->part_cap = need;
  }
  d.part = net->part;
  for (int l = 1; l <= L; ++l) {
    DwLayer& q = d.l[l - 1];
    q.dZ = net->dZ[l];
    q.H = l == 1 ? X : net->H[l - 1];
    q.M = net->sizes[l];
    q.N = net->sizes[l - 1];
    q.Np = round16(q.N);
    q.mtiles = (q.M + FM - 1) / FM;
    q.first = d.blocks;
    q.poff = net->woff[l - 1];
    q.boff = net->boff[l - 1];
    d.blocks += q.mtiles * d.slices;
  }
  MCK(cudaFuncSetAttribute(k_mlp_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dw_smem()));
  k_mlp_dw<<<d.blocks, DW_THREADS, dw_smem(), net->stream>>>(d);
  MCK(cudaGetLastError());
  k_mlp_dw_sum<<<(unsigned)((net->nparam + 255) / 256), 256, 0, net->stream>>>(net->nparam, d.slices, d.part, d.g);
  MCK(cudaGetLastError());
  return YTF_OK;
}

// after a synchronisation: a tensor-core wait that ran out in the work before it
int check_waits(ytf_mlp* net) {
  if (!*net->tc_err) return YTF_OK;
  *net->tc_err = 0;
  return mfail(net, YTF_ERR_CUDA, "ytf_mlp: a tensor-core pipeline wait timed out");
}

// forward pass of B samples already in H[0]
int forward(ytf_mlp* net, int B) {
  const int L = (int)net->sizes.size() - 1;
  const long n = net->nparam;
  k_to_bf16<<<(unsigned)((n + 255) / 256), 256, 0, net->stream>>>(n, net->p, net->wb);
  MCK(cudaGetLastError());
  for (int l = 1; l <= L; ++l) {
    const int in = net->sizes[l - 1], out = net->sizes[l];
    MCK((gemm<float, __nv_bfloat16>(net, B, out, in, net->H[l - 1], in, 1, net->wb + net->woff[l - 1], 1, in,
                                   net->Z[l], out, net->p + net->boff[l - 1], net->H[l], l < L ? 1 : 0, 0)));
  }
  return YTF_OK;
}

// backward from the targets in T; gradients into g
int backward(ytf_mlp* net, int B) {
  const int L = (int)net->sizes.size() - 1;
  k_loss<<<(B + 255) / 256, 256, 0, net->stream>>>(B, net->H[L], net->T, net->dZ[L], net->lb);
  MCK(cudaGetLastError());
  for (int l = L; l >= 1; --l) {
    const int in = net->sizes[l - 1], out = net->sizes[l];
    if (l < L) {
      const long cnt = (long)B * out;
      k_gelu_back<<<(unsigned)((cnt + 255) / 256), 256, 0, net->stream>>>(cnt, net->Z[l], net->dH[l], net->dZ[l]);
      MCK(cudaGetLastError());
    }
    // dW = dZ^T H, db = Σ dZ
    MCK((gemm<float, float>(net, out, in, B, net->dZ[l], 1, out, net->H[l - 1], in, 1, net->g + net->woff[l - 1],
                           in, nullptr, nullptr, 0, 0)));
    k_colsum<<<(out + 255) / 256, 256, 0, net->stream>>>(B, out, net->dZ[l], net->g + net->boff[l - 1]);
    MCK(cudaGetLastError());
    if (l > 1)
      MCK((gemm<float, __nv_bfloat16>(net, B, in, out, net->dZ[l], out, 1, net->wb + net->woff[l - 1], in, 1,
                                     net->dH[l - 1], in, nullptr, nullptr, 0, 0)));
  }
  return YTF_OK;
}

// loss terms into lb and gradients into g of the batch in H[0], T
int loss_and_gradients(ytf_mlp* net, int B) {
  int rc;
  if (!net->fused) {
    if ((rc = forward(net, B))) return rc;
    return backward(net, B);
  }
  if ((rc = pack_weights(net, true)) || (rc = forward_fused(net, B, net->H[0], net->H[net->sizes.size() - 1], true)))
    return rc;
  return backward_fused(net, B, net->H[0]);
}

}  // namespace

extern "C" {

int ytf_mlp_create(int device, int nlayers, const int* sizes, unsigned long long seed, ytf_mlp** out) {
  if (!out || nlayers < 1 || !sizes) return YTF_ERR_ARG;
  *out = nullptr;
  for (int l = 0; l <= nlayers; ++l)
    if (sizes[l] < 1) return YTF_ERR_ARG;
  if (sizes[nlayers] != 2) return YTF_ERR_ARG;  // (log-response, pole-score logit)
  if (cudaSetDevice(device) != cudaSuccess) return YTF_ERR_CUDA;
  ytf_mlp* net = new ytf_mlp();
  net->device = device;
  net->sizes.assign(sizes, sizes + nlayers + 1);
  long o = 0;
  for (int l = 1; l <= nlayers; ++l) {
    net->woff.push_back(o);
    o += (long)sizes[l] * sizes[l - 1];
    net->boff.push_back(o);
    o += sizes[l];
  }
  net->nparam = o;
  // He-style initialisation from a seeded 64-bit LCG (uniform, variance 2 / fan_in), zero bias
  std::vector<float> h(o, 0.f);
  unsigned long long st = seed * 6364136223846793005ull + 1442695040888963407ull;
  for (int l = 1; l <= nlayers; ++l) {
    const float a = std::sqrt(6.0f / sizes[l - 1]) * (l == nlayers ? 0.5f : 1.0f);
    for (long i = 0; i < (long)sizes[l] * sizes[l - 1]; ++i) {
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      const double u = (double)(st >> 11) * (1.0 / 9007199254740992.0);
      h[net->woff[l - 1] + i] = (float)((2 * u - 1) * a);
    }
  }
  int rc = YTF_OK;
  if (cudaMalloc(&net->p, 4 * o) != cudaSuccess || cudaMalloc(&net->g, 4 * o) != cudaSuccess ||
      cudaMalloc(&net->m, 4 * o) != cudaSuccess || cudaMalloc(&net->v, 4 * o) != cudaSuccess ||
      cudaMalloc(&net->wb, 2 * o) != cudaSuccess ||
      cudaHostAlloc(&net->tc_err, sizeof(unsigned), cudaHostAllocDefault) != cudaSuccess)
    rc = YTF_ERR_NOMEM;
  else
    *net->tc_err = 0;
  cudaDeviceGetAttribute(&net->nsm, cudaDevAttrMultiProcessorCount, device);
  net->fused = nlayers <= FMAXL;
  for (int l = 0; l <= nlayers; ++l) net->fused = net->fused && sizes[l] <= FW;
  if (!rc && net->fused) {
    size_t bytes = 0;
    for (int trans = 0; trans < 2; ++trans)
      for (int l = 1; l <= nlayers; ++l) {
        const int rows = trans ? sizes[l - 1] : sizes[l], k = trans ? sizes[l] : sizes[l - 1];
        (trans ? net->img_b : net->img_f).push_back(bytes);
        bytes += 2ul * round16(rows) * 64 * ((k + FKB - 1) / FKB);
      }
    if (cudaMalloc(&net->img, bytes) != cudaSuccess) rc = YTF_ERR_NOMEM;
  }
  if (!rc && (cudaMemcpy(net->p, h.data(), 4 * o, cudaMemcpyHostToDevice) != cudaSuccess ||
              cudaMemset(net->m, 0, 4 * o) != cudaSuccess || cudaMemset(net->v, 0, 4 * o) != cudaSuccess ||
              cudaMemset(net->g, 0, 4 * o) != cudaSuccess))
    rc = YTF_ERR_CUDA;
  if (rc) { delete net; return rc; }
  *out = net;
  return YTF_OK;
}

int ytf_mlp_destroy(ytf_mlp* net) {
  if (net) { cudaSetDevice(net->device); cudaStreamSynchronize(net->stream); delete net; }
  return YTF_OK;
}

const char* ytf_mlp_last_error(const ytf_mlp* net) { return net ? net->err.c_str() : "null network"; }

long ytf_mlp_num_params(const ytf_mlp* net) { return net ? net->nparam : 0; }

int ytf_mlp_set_stream(ytf_mlp* net, void* stream) {
  if (!net) return YTF_ERR_ARG;
  net->stream = (cudaStream_t)stream;
  return YTF_OK;
}

int ytf_mlp_params(ytf_mlp* net, float* get, const float* set) {
  if (!net) return YTF_ERR_ARG;
  MCK(cudaSetDevice(net->device));
  if (set) MCK(cudaMemcpyAsync(net->p, set, 4 * net->nparam, cudaMemcpyHostToDevice, net->stream));
  if (get) MCK(cudaMemcpyAsync(get, net->p, 4 * net->nparam, cudaMemcpyDeviceToHost, net->stream));
  MCK(cudaStreamSynchronize(net->stream));
  return YTF_OK;
}

int ytf_mlp_forward(ytf_mlp* net, int B, const float* X, float* out, int on_device) {
  if (!net || B < 0 || (B > 0 && (!X || !out))) return YTF_ERR_ARG;
  if (B == 0) return YTF_OK;
  MCK(cudaSetDevice(net->device));
  int rc;
  const size_t xb = sizeof(float) * B * net->sizes[0];
  if (net->fused) {
    // device memory is used where it lies, unless it is another GPU's or the outputs lie over the inputs (a CTA
    // writes its rows' outputs while others still read)
    const uintptr_t x0 = (uintptr_t)X, y0 = (uintptr_t)out;
    const bool overlap = x0 < y0 + sizeof(float) * 2 * B && y0 < x0 + xb;
    const bool xcopy = !on_device || overlap || other_device(net->device, X);
    const bool ycopy = !on_device || other_device(net->device, out);
    if ((xcopy || ycopy) && (rc = ensure_io(net, B))) return rc;
    if (xcopy)
      MCK(cudaMemcpyAsync(net->Xin, X, xb, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, net->stream));
    float* y = ycopy ? net->Yout : out;
    if ((rc = pack_weights(net, false)) || (rc = forward_fused(net, B, xcopy ? net->Xin : X, y, false))) return rc;
    if (ycopy)
      MCK(cudaMemcpyAsync(out, y, sizeof(float) * 2 * B, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                          net->stream));
    MCK(cudaStreamSynchronize(net->stream));
    return check_waits(net);
  }
  rc = ensure(net, B);
  if (rc) return rc;
  MCK(cudaMemcpyAsync(net->H[0], X, xb, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, net->stream));
  if ((rc = forward(net, B))) return rc;
  const int L = (int)net->sizes.size() - 1;
  MCK(cudaMemcpyAsync(out, net->H[L], sizeof(float) * 2 * B, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                      net->stream));
  MCK(cudaStreamSynchronize(net->stream));
  return check_waits(net);
}

int ytf_mlp_gradients(ytf_mlp* net, int B, const float* X, const float* T, float* grad, float* loss, int on_device) {
  if (!net || B < 1 || !X || !T) return YTF_ERR_ARG;
  MCK(cudaSetDevice(net->device));
  int rc = ensure(net, B);
  if (rc) return rc;
  const auto kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  MCK(cudaMemcpyAsync(net->H[0], X, sizeof(float) * B * net->sizes[0], kind, net->stream));
  MCK(cudaMemcpyAsync(net->T, T, sizeof(float) * 2 * B, kind, net->stream));
  if ((rc = loss_and_gradients(net, B))) return rc;
  if (grad) MCK(cudaMemcpyAsync(grad, net->g, 4 * net->nparam, cudaMemcpyDeviceToHost, net->stream));
  if (loss) {
    std::vector<float> lb(B);
    MCK(cudaMemcpyAsync(lb.data(), net->lb, 4 * (size_t)B, cudaMemcpyDeviceToHost, net->stream));
    MCK(cudaStreamSynchronize(net->stream));
    double s = 0;
    for (float x : lb) s += x;
    *loss = (float)(s / B);
  }
  MCK(cudaStreamSynchronize(net->stream));
  return check_waits(net);
}

int ytf_mlp_train(ytf_mlp* net, long n, const float* X, const float* T, int batch, int steps, float lr,
                  unsigned long long seed, float* losses) {
  if (!net || n < 1 || !X || !T || batch < 1 || steps < 0) return YTF_ERR_ARG;
  MCK(cudaSetDevice(net->device));
  int rc = ensure(net, batch);
  if (rc) return rc;
  const int d = net->sizes[0];
  // mini-batches drawn from the device-resident set (X: [n][d], T: [n][2]) on the device
  float* dl = nullptr;
  MCK(cudaMalloc(&dl, sizeof(float) * batch));
  std::vector<float> lb(batch);
  for (int s = 0; s < steps; ++s) {
    const long cnt = (long)batch * (d + 2);
    k_gather<<<(unsigned)((cnt + 255) / 256), 256, 0, net->stream>>>(batch, d, n, seed, net->step, X, T, net->H[0],
                                                                      net->T);
    if (cudaGetLastError() != cudaSuccess) { cudaFree(dl); return mfail(net, YTF_ERR_CUDA, "gather launch"); }
    if ((rc = loss_and_gradients(net, batch))) { cudaFree(dl); return rc; }
    net->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)net->step), c2 = 1.f - std::pow(b2, (float)net->step);
    k_adam<<<(unsigned)((net->nparam + 255) / 256), 256, 0, net->stream>>>(net->nparam, net->p, net->g, net->m, net->v,
                                                                           lr, b1, b2, 1e-8f, c1, c2);
    if (cudaGetLastError() != cudaSuccess) { cudaFree(dl); return mfail(net, YTF_ERR_CUDA, "adam launch"); }
    if (losses) {
      cudaMemcpyAsync(lb.data(), net->lb, 4 * (size_t)batch, cudaMemcpyDeviceToHost, net->stream);
      cudaStreamSynchronize(net->stream);
      double a = 0;
      for (float x : lb) a += x;
      losses[s] = (float)(a / batch);
    }
  }
  cudaFree(dl);
  MCK(cudaStreamSynchronize(net->stream));
  return check_waits(net);
}

}  // extern "C"

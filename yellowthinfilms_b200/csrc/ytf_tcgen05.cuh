// ytf_tcgen05.cuh -- small inline-PTX wrappers for the sm_100a tensor-core kernels:
// shared-memory matrix descriptors (canonical K-major, no swizzle), mbarrier operations,
// one-dimensional bulk copies, tcgen05 commit/fences and tcgen05.ld of 32-bit columns.
#pragma once
#include <cstdint>

namespace ytf {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of (row r, K byte kb) in a plane of 64-byte rows: [R/8][4 K-cores][8 rows][16 B]
__device__ __forceinline__ uint32_t plane_off(int r, int kb) {
  return (uint32_t)((r >> 3) * 512 + (kb >> 4) * 128 + (r & 7) * 16 + (kb & 15));
}

// 1.5 2^52 + 0x808080: the low word of fma(v, scale, AI_MAGIC) is rint(v scale) + 0x808080, whose bytes are
// the balanced digits + 128
constexpr double AI_MAGIC = 6755399441055744.0 + 8421504.0;
// the same of the rounded product: rint(fl(v scale)) + 0x808080
__device__ __forceinline__ uint32_t fixed_bits(double v, double scale) {
  return (uint32_t)__double2loint(__dadd_rn(__dmul_rn(v, scale), AI_MAGIC));
}
// the digit planes (most significant first) of four such words, one byte each: seven byte permutes in
// place of the shifts, masks and additions of every digit by itself
__device__ __forceinline__ void digit_words(const uint32_t u[4], uint32_t& d0, uint32_t& d1, uint32_t& d2) {
  const uint32_t l01 = __byte_perm(u[0], u[1], 0x5140), l23 = __byte_perm(u[2], u[3], 0x5140);
  const uint32_t h01 = __byte_perm(u[0], u[1], 0x0062), h23 = __byte_perm(u[2], u[3], 0x0062);
  d0 = __byte_perm(h01, h23, 0x5410) ^ 0x80808080u;
  d1 = __byte_perm(l01, l23, 0x7632) ^ 0x80808080u;
  d2 = __byte_perm(l01, l23, 0x5410) ^ 0x80808080u;
}

// shared-memory matrix descriptor: start >> 4, LBO = 128 B (the two K-cores of one MMA),
// SBO = 512 B (consecutive 8-row groups), descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(512u >> 4) << 32) |
         (1ull << 46);
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(addr), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void mbar_init(uint32_t addr, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint32_t addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(addr), "r"(bytes) : "memory");
}

// one-dimensional bulk copy global -> this CTA's shared memory, completion counted in bytes on
// an mbarrier (no multicast; addresses 16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t ta, uint32_t v[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(ta)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

}  // namespace ytf

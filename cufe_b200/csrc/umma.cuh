// umma.cuh -- the fifth-generation tensor core for exact integer products: tcgen05.mma kind::i8
// (8-bit operands from shared memory, 32-bit integer accumulators in TMEM), its descriptors,
// completion barriers and accumulator loads.
//
// Operands are K-major without swizzle: rows of K bytes cut into core matrices of 8 rows x 16
// bytes (128 contiguous bytes); `lbo` is the byte distance of neighbouring core matrices along K,
// the 8-row groups along M or N are 128 bytes apart.
#pragma once
#include "cufe_internal.cuh"

namespace cufe {

// A barrier wait gives up after this many tries of at most a microsecond each; a correct launch
// waits microseconds.
constexpr uint32_t kUmmaWaitLimit = 1u << 20;

__device__ __forceinline__ uint32_t smem_u32_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) | ((uint64_t)(128u >> 4) << 32) |
         (1ull << 46);
}

// M = 128 rows of A (signed or unsigned bytes) by n rows of B (unsigned bytes), s32 accumulators
__host__ __device__ constexpr uint32_t umma_i8_desc(bool a_signed, uint32_t n) {
  return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// D[tmem] (+)= A B for 32 bytes of K; one thread issues it
__device__ __forceinline__ void umma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  const uint32_t zero = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate), "r"(zero)
      : "memory");
}
// arrives at `bar` when every umma issued by this thread so far has completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// columns (a power of two >= 32) of TMEM; one whole warp; the address lands at shared `slot`
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns));
}
__device__ __forceinline__ void umma_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// this thread's shared-memory writes become visible to the tensor core's reads
__device__ __forceinline__ void smem_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 8 accumulator columns of the warp's 32 TMEM lanes (the warp's quarter: warp index mod 4), one
// lane per thread; valid after tmem_wait_ld
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// zeroes 8 columns of the warp's 32 TMEM lanes; complete after tmem_wait_st
__device__ __forceinline__ void tmem_zero8(uint32_t addr) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(addr), "r"(0u)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// waits for the completion of the phase with this parity; false when it gave up
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < kUmmaWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000u)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// announces `bytes` of bulk copies that will complete on `bar`, and arrives
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// `bytes` (a multiple of 16) from global memory to shared memory, both 16-byte aligned
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
               : "memory");
}

// 4 x 4 byte transpose: out[b] = bytes b of w[0..3], w[0]'s lowest
__device__ __forceinline__ void byte_transpose(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t (&o)[4]) {
  const uint32_t a = __byte_perm(w0, w1, 0x5140), b = __byte_perm(w2, w3, 0x5140);  // bytes 0, 1 interleaved
  const uint32_t c = __byte_perm(w0, w1, 0x7362), d = __byte_perm(w2, w3, 0x7362);  // bytes 2, 3
  o[0] = __byte_perm(a, b, 0x5410);
  o[1] = __byte_perm(a, b, 0x7632);
  o[2] = __byte_perm(c, d, 0x5410);
  o[3] = __byte_perm(c, d, 0x7632);
}

}  // namespace cufe

// aes.cuh -- AES-256 block function for the samplers' keystreams (FIPS-197).
//
// T-table formulation (one SubBytes+ShiftRows+MixColumns round = 16 table lookups + XORs).
// Each of the four 256-entry tables is replicated once per shared-memory bank so a warp's 32
// lookups never conflict: entry x of table t for lane L lives at the shared-memory address
//   0x10000 + (t >> 1) * 64 KiB + x * 256 + (t & 1) * 128 + L * 4,
// so the lookup address is one PRMT of the state word with the per-lane constant 0x100 | L * 4
// (the table offset is an immediate of the LDS).  The fixed address makes the base part of that
// constant: relative to the base of the dynamic shared memory, which only the linker knows, the
// compiler spent one more addition per lookup whenever its address folding did not apply (1,411
// against 1,039 million instructions for the sigma_3 candidates of four encryptions at n = 4096,
// l = 784).  Kernels that use the tables therefore take kAesSmemBytes = 192 KiB of dynamic
// shared memory and no static one of 64 KiB; it starts below address 0x10000 then, so it covers the tables,
// which every such kernel checks before it writes them.
// Round keys are 60 big-endian words in registers; an all-zero key schedule is valid (the
// reference CPU path's uninitialised AES contexts).
#pragma once
#include "cufe_internal.cuh"

namespace cufe {

constexpr uint32_t kAesTables = 0x10000;     // shared-memory address of the tables
constexpr int kAesTableBytes = 131072;
constexpr int kAesSmemBytes = (int)kAesTables + kAesTableBytes;  // dynamic shared memory of a kernel with tables

// S-box, uploaded by sampler_init_device (computed from GF(2^8) inversion + affine map)
static __constant__ uint8_t c_sbox[256];

__device__ __forceinline__ uint32_t xtime_u8(uint32_t b) {
  return ((b << 1) ^ ((b & 0x80u) ? 0x1bu : 0u)) & 0xffu;
}

// whether dynamic shared memory of `bytes` from address `base` holds the tables
__host__ __device__ constexpr bool aes_tables_fit(uint32_t base, uint32_t bytes) {
  return base <= kAesTables && bytes >= (uint32_t)kAesTableBytes && base + bytes - kAesTableBytes >= kAesTables;
}
static_assert(aes_tables_fit(0, kAesSmemBytes) && aes_tables_fit(0x400, kAesSmemBytes) &&
                  aes_tables_fit(kAesTables, kAesSmemBytes) && aes_tables_fit(kAesTables, kAesTableBytes),
              "tables inside");
static_assert(!aes_tables_fit(kAesTables + 1, kAesSmemBytes) && !aes_tables_fit(0, kAesSmemBytes - 1) &&
                  !aes_tables_fit(0x400, kAesTableBytes) && !aes_tables_fit(0, 0),
              "tables outside");

// fill the replicated tables (all threads of the CTA, a multiple of 16; caller syncs): 16 threads
// write the 256 bytes of one entry of a pair of tables, 16 bytes each.  False, with nothing written and
// the status set, where the CTA's shared memory does not lie as they need it.
__device__ __forceinline__ bool aes_fill_tables(uint32_t *status) {
  extern __shared__ uint32_t smem_u32[];
  uint32_t bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(bytes));
  if (!aes_tables_fit((uint32_t)__cvta_generic_to_shared(smem_u32), bytes)) {
    if (threadIdx.x == 0) atomicOr(status, kStatusAesTables);
    return false;
  }
  const uint32_t tid = threadIdx.x + threadIdx.y * blockDim.x, piece = tid & 15u;
  for (uint32_t x = tid >> 4; x < 256; x += (blockDim.x * blockDim.y) >> 4) {
    const uint32_t s = c_sbox[x], d = xtime_u8(s);
    const uint32_t te0 = (d << 24) | (s << 16) | (s << 8) | (d ^ s);
    const uint32_t lo = piece & 8u ? __funnelshift_r(te0, te0, 8) : te0, hi = __funnelshift_r(lo, lo, 16);
    const uint32_t at = kAesTables + x * 256 + piece * 16;
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(lo) : "memory");
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at + 65536), "r"(hi) : "memory");
  }
  return true;
}

struct AesCtx {
  uint32_t laneoff;  // (kAesTables >> 8) | (lane & 31) * 4
};
__device__ __forceinline__ AesCtx aes_ctx() { return AesCtx{(kAesTables >> 8) | ((threadIdx.x & 31u) * 4u)}; }

template <int T>
__device__ __forceinline__ uint32_t te(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1 + %2];" : "=r"(v) : "r"(addr), "n"((T >> 1) * 65536 + (T & 1) * 128));
  return v;
}
// byte b (3 = most significant) of s as a table address: bytes (0, kAesTables >> 16, b, lane * 4)
template <int B>
__device__ __forceinline__ uint32_t taddr(AesCtx c, uint32_t s) {
  return __byte_perm(s, c.laneoff, 0x6504 | (B << 4));
}

// rounds R0..13 on the state after round R0 - 1 (R0 = 1: after the initial AddRoundKey)
template <int R0>
__device__ __forceinline__ void aes256_inner_rounds(uint32_t &s0, uint32_t &s1, uint32_t &s2, uint32_t &s3,
                                                    const uint32_t (&rk)[60], AesCtx c) {
#pragma unroll
  for (int r = R0; r < 14; ++r) {
    const uint32_t t0 = te<0>(taddr<3>(c, s0)) ^ te<1>(taddr<2>(c, s1)) ^
                        te<2>(taddr<1>(c, s2)) ^ te<3>(taddr<0>(c, s3)) ^ rk[4 * r];
    const uint32_t t1 = te<0>(taddr<3>(c, s1)) ^ te<1>(taddr<2>(c, s2)) ^
                        te<2>(taddr<1>(c, s3)) ^ te<3>(taddr<0>(c, s0)) ^ rk[4 * r + 1];
    const uint32_t t2 = te<0>(taddr<3>(c, s2)) ^ te<1>(taddr<2>(c, s3)) ^
                        te<2>(taddr<1>(c, s0)) ^ te<3>(taddr<0>(c, s1)) ^ rk[4 * r + 2];
    const uint32_t t3 = te<0>(taddr<3>(c, s3)) ^ te<1>(taddr<2>(c, s0)) ^
                        te<2>(taddr<1>(c, s1)) ^ te<3>(taddr<0>(c, s2)) ^ rk[4 * r + 3];
    s0 = t0;
    s1 = t1;
    s2 = t2;
    s3 = t3;
  }
}

// (a & m) | (b & ~m)
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t b, uint32_t m) { return (a & m) | (b & ~m); }

// one word of the final round: S-box bytes 3..0 of a, b, d, e (taken from the tables: Te2 byte 3,
// Te3 byte 2, Te0 byte 1, Te1 byte 0) with round key k
__device__ __forceinline__ uint32_t aes256_last(AesCtx c, uint32_t a, uint32_t b, uint32_t d, uint32_t e,
                                                uint32_t k) {
  const uint32_t hi = bit_select(te<2>(taddr<3>(c, a)), te<3>(taddr<2>(c, b)), 0xff000000u);
  const uint32_t lo = bit_select(te<0>(taddr<1>(c, d)), te<1>(taddr<0>(c, e)), 0x0000ff00u);
  return bit_select(hi, lo, 0xffff0000u) ^ k;
}

// rounds R0..14 on the state after round R0 - 1
template <int R0>
__device__ __forceinline__ void aes256_rounds_from(uint32_t &s0, uint32_t &s1, uint32_t &s2, uint32_t &s3,
                                                   const uint32_t (&rk)[60], AesCtx c) {
  aes256_inner_rounds<R0>(s0, s1, s2, s3, rk, c);
  const uint32_t o0 = aes256_last(c, s0, s1, s2, s3, rk[56]), o1 = aes256_last(c, s1, s2, s3, s0, rk[57]);
  const uint32_t o2 = aes256_last(c, s2, s3, s0, s1, rk[58]), o3 = aes256_last(c, s3, s0, s1, s2, rk[59]);
  s0 = o0;
  s1 = o1;
  s2 = o2;
  s3 = o3;
}

// rounds 1..14 on a state that already holds input ^ rk[0..3]
__device__ __forceinline__ void aes256_rounds(uint32_t &s0, uint32_t &s1, uint32_t &s2, uint32_t &s3,
                                              const uint32_t (&rk)[60], AesCtx c) {
  aes256_rounds_from<1>(s0, s1, s2, s3, rk, c);
}

// Counter caching for the CPU mapping with nonce 0: the input block is 0^12 || BE32(ctr), so
// after the initial AddRoundKey only state word 3 depends on ctr.  In round 1 each output
// word takes exactly one byte of word 3 (T3 of its low byte for word 0, T2/T1/T0 of the
// higher bytes for words 1..3); for counters with equal upper 24 bits, words 1..3 after round
// 1 are therefore fixed and only word 0 varies, and in round 2 each output word takes one byte
// of word 0 and three fixed bytes.  k0, k1: the ctr-independent part of words 0 and 1 after round
// 1 (per key); d0..d3: what words 2 and 3 give to round 2, fixed for counters with equal upper
// 16 bits; c0..c3: that and word 1's share, fixed for equal upper 24 bits (`hi`).  Per block, rounds
// 1 and 2 then take 1 + 4 table lookups instead of 32, and 5 more when `hi` changes.  d0..d3
// change every 65,536 counters (2,730 refills), so what only they need is read from the key
// schedule in global memory (rkg).
struct CtrCache {
  uint32_t k0, k1, d0, d1, d2, d3, c0, c1, c2, c3, hi;
};

__device__ __forceinline__ void ctr_cache_key(CtrCache &cc, const uint32_t (&rk)[60], AesCtx c) {
  const uint32_t s0 = rk[0], s1 = rk[1], s2 = rk[2];
  cc.k0 = te<0>(taddr<3>(c, s0)) ^ te<1>(taddr<2>(c, s1)) ^ te<2>(taddr<1>(c, s2)) ^ rk[4];
  cc.k1 = te<0>(taddr<3>(c, s1)) ^ te<1>(taddr<2>(c, s2)) ^ te<3>(taddr<0>(c, s0)) ^ rk[5];
  cc.hi = 0xffffffffu;  // no counter cached
}

// d0..d3 for the counters with the upper 16 bits of ctr
__device__ __noinline__ uint4 ctr_cache_upper(uint32_t ctr, const uint32_t *__restrict__ rkg, AesCtx c) {
  const uint4 a = __ldg(reinterpret_cast<const uint4 *>(rkg)), b = __ldg(reinterpret_cast<const uint4 *>(rkg + 4));
  const uint4 k = __ldg(reinterpret_cast<const uint4 *>(rkg + 8));
  const uint32_t w3 = ctr ^ a.w;
  const uint32_t u2 = te<0>(taddr<3>(c, a.z)) ^ te<1>(taddr<2>(c, w3)) ^ te<2>(taddr<1>(c, a.x)) ^
                      te<3>(taddr<0>(c, a.y)) ^ b.z;
  const uint32_t u3 = te<0>(taddr<3>(c, w3)) ^ te<1>(taddr<2>(c, a.x)) ^ te<2>(taddr<1>(c, a.y)) ^
                      te<3>(taddr<0>(c, a.z)) ^ b.w;
  return make_uint4(te<2>(taddr<1>(c, u2)) ^ te<3>(taddr<0>(c, u3)) ^ k.x,
                    te<1>(taddr<2>(c, u2)) ^ te<2>(taddr<1>(c, u3)) ^ k.y,
                    te<0>(taddr<3>(c, u2)) ^ te<1>(taddr<2>(c, u3)) ^ k.z,
                    te<0>(taddr<3>(c, u3)) ^ te<3>(taddr<0>(c, u2)) ^ k.w);
}

// the keystream block of counter ctr (nonce 0), output as in aes256_ctr_block; rkg: the same
// key schedule as rk, in global memory.  `even`, `odd`
// (warp-uniform): whether words 0, 2 and words 1, 3 are wanted; the other pair is left out of the
// final round (8 of its 16 lookups) and 0 in o.
__device__ __forceinline__ void aes256_ctr_block_cached(uint32_t (&o)[4], uint32_t ctr, const uint32_t (&rk)[60],
                                                        const uint32_t *__restrict__ rkg, AesCtx c, CtrCache &cc,
                                                        bool even, bool odd) {
  const uint32_t w3 = ctr ^ rk[3];
  if ((ctr >> 8) != cc.hi) {
    if (((ctr >> 8) ^ cc.hi) >> 8) {
      const uint4 d = ctr_cache_upper(ctr, rkg, c);
      cc.d0 = d.x;
      cc.d1 = d.y;
      cc.d2 = d.z;
      cc.d3 = d.w;
    }
    cc.hi = ctr >> 8;
    const uint32_t u1 = cc.k1 ^ te<2>(taddr<1>(c, w3));
    cc.c0 = cc.d0 ^ te<1>(taddr<2>(c, u1));
    cc.c1 = cc.d1 ^ te<0>(taddr<3>(c, u1));
    cc.c2 = cc.d2 ^ te<3>(taddr<0>(c, u1));
    cc.c3 = cc.d3 ^ te<2>(taddr<1>(c, u1));
  }
  const uint32_t a0 = cc.k0 ^ te<3>(taddr<0>(c, w3));
  uint32_t s0 = cc.c0 ^ te<0>(taddr<3>(c, a0)), s1 = cc.c1 ^ te<3>(taddr<0>(c, a0));
  uint32_t s2 = cc.c2 ^ te<2>(taddr<1>(c, a0)), s3 = cc.c3 ^ te<1>(taddr<2>(c, a0));
  aes256_inner_rounds<3>(s0, s1, s2, s3, rk, c);
  o[0] = o[1] = o[2] = o[3] = 0;
  if (even) {
    o[0] = aes256_last(c, s0, s1, s2, s3, rk[56]);
    o[2] = aes256_last(c, s2, s3, s0, s1, rk[58]);
  }
  if (odd) {
    o[1] = aes256_last(c, s1, s2, s3, s0, rk[57]);
    o[3] = aes256_last(c, s3, s0, s1, s2, rk[59]);
  }
}

// One keystream block of the CPU counter mapping (src/aes256ctr.c:13-81): input
// BE16(nonce) || 0^10 || BE32(ctr); output as four big-endian words.
__device__ __forceinline__ void aes256_ctr_block(uint32_t (&o)[4], uint32_t nonce_word, uint32_t ctr,
                                                 const uint32_t (&rk)[60], AesCtx c) {
  uint32_t s0 = nonce_word ^ rk[0], s1 = rk[1], s2 = rk[2], s3 = ctr ^ rk[3];
  aes256_rounds(s0, s1, s2, s3, rk, c);
  o[0] = s0;
  o[1] = s1;
  o[2] = s2;
  o[3] = s3;
}

__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

}  // namespace cufe

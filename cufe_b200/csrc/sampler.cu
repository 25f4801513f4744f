// sampler.cu -- AES-256-CTR keystreams and the discrete Gaussian / uniform samplers.
//
// Two counter-to-sample mappings are implemented, both bit-exact:
//
//  * CPU mapping (src/gauss.c + src/aes256ctr.c): one AES-CTR stream per context; every
//    gaussian_sampler_* call consumes 384-byte refills (24 counter blocks) in order, takes
//    the accepted candidates in order and drops the rest of its last refill.  The stream is
//    sequential by construction, so it is computed in three parallel phases: (1) every
//    refill's 8 candidates and accept mask for a generous refill range (the AES work, one
//    thread per refill), (2) a per-stream exclusive scan of accept counts and a one-warp
//    walk that finds where each call starts (each call starts at a fresh refill), (3) a
//    scatter of the accepted candidates to their coefficient positions as residues.
//  * GPU mapping (src/sample_gpu.cu, src/AES.cuh): thread t of polynomial p owns coefficients
//    8t..8t+7 and draws chained-AES refills from counter p*5*T*24 + rep*T*24 + t*24.
#include "aes.cuh"
#include "sampler.cuh"
#include "sampler_host.h"
#include "scheme.cuh"
#include "prof.h"

#include <algorithm>
#include <cmath>

namespace cufe {

namespace {

__device__ __forceinline__ uint64_t le64_of(uint32_t be_lo, uint32_t be_hi) {
  return (uint64_t)bswap32(be_lo) | ((uint64_t)bswap32(be_hi) << 32);
}

// ------------------------------------------------------------------ CPU mapping, phase 1

// one keystream block of the CPU mapping from round keys in global memory (rare paths)
__device__ __noinline__ void ctr_block_g(uint32_t (&W)[4], uint32_t ctr, const uint32_t *__restrict__ rkg,
                                         AesCtx c) {
  uint32_t rk[60];
#pragma unroll
  for (int i = 0; i < 60; ++i) rk[i] = __ldg(rkg + i);
  aes256_ctr_block(W, 0u, ctr, rk, c);
}

// uniform draws when the first 10 words hold fewer than 8 accepted ones (at least 3 of 10
// draws rejected: about 7e-5 per refill for sigma_2 and sigma_3, whose rejection rate is
// 1 - 7 K / 2^32 = 0.84%; far less for sigma_1): rescan bytes 200.. with the rejection loop of
// src/gauss.c:578-703, regenerating blocks as needed
template <int SIG>
__device__ __noinline__ void uniform_slow(uint32_t *y, int ystride, uint32_t cb, const uint32_t *__restrict__ rkg,
                                          AesCtx c, uint32_t *status) {
  int w = 0, have_blk = -1;
  uint32_t W[4] = {0, 0, 0, 0};
  for (int j = 0; j < 8; ++j) {
    uint32_t x = 0;
    for (;;) {
      if (w >= 46) {  // would read beyond the 384-byte refill: undefined in the reference
        atomicOr(status, kStatusUniformOverrun);
        x = 0;
        break;
      }
      const int byte = 200 + 4 * w, blk = byte >> 4;
      if (blk != have_blk) {
        ctr_block_g(W, cb + (uint32_t)blk, rkg, c);
        have_blk = blk;
      }
      const int wi = (byte >> 2) & 3;
      x = bswap32(wi == 0 ? W[0] : wi == 1 ? W[1] : wi == 2 ? W[2] : W[3]);
      ++w;
      if (uniform_ok<SIG>(x)) break;
    }
    y[j * ystride] = uniform_reduce<SIG>(x);
  }
}

// keystream word w (bytes 4w..4w+3, little-endian) of a refill
__device__ __forceinline__ uint32_t refill_word(int w, uint32_t cb, const uint32_t *__restrict__ rkg,
                                                AesCtx c) {
  uint32_t W[4];
  ctr_block_g(W, cb + (uint32_t)(w >> 2), rkg, c);
  const int i = w & 3;
  return bswap32(i == 0 ? W[0] : i == 1 ? W[1] : i == 2 ? W[2] : W[3]);
}

// What a refill keeps of candidate ln beside z's low word: its accept bit (bit ln), bit 32 of z (bit
// 8 + ln; |value| = z < 8K < 2^33), and bit 16 if an accepted z ever reaches 2^33.
__device__ __forceinline__ uint32_t candidate_bits(int ln, bool b, uint64_t z, uint32_t k8) {
  const uint32_t a = accept_final(b, z, (k8 >> ln) & 1u);
  return (a << ln) | ((uint32_t)((z >> 32) & 1u) << (8 + ln)) | ((a & (uint32_t)((z >> 33) != 0)) << 16);
}

// The candidates of a refill that its top words left undecided (bits of `open`), again from their
// full words: CDT words 8 + 2 lane, 9 + 2 lane and, for the 126-bit compare of the CPU S3, 2 lane, 1
// + 2 lane; Bernoulli words 16 + 2 lane, 17 + 2 lane; exponent bytes in word 24 (all 25 words
// further for lanes 4..7).  Rewrites their low words in cand[8] and returns `bits` with theirs
// corrected.
template <int SIG, bool FULL, int VAR>
__device__ __noinline__ uint32_t refill_slow(uint32_t open, uint32_t k8, uint32_t cb,
                                             const uint32_t *__restrict__ rkg, AesCtx c, double kinv,
                                             uint32_t *cand, uint32_t bits, uint32_t *status) {
  uint32_t y[8];
  uniform_slow<SIG>(y, 1, cb, rkg, c, status);
  for (; open; open &= open - 1) {
    const int ln = __ffs(open) - 1, w = (ln < 4 ? 0 : 25) + 2 * (ln & 3);
    uint64_t v[3];  // r1, r2, rm
#pragma unroll 1
    for (int i = 0; i < 3; ++i)
      v[i] = refill_word(w + 8 * i, cb, rkg, c) | ((uint64_t)refill_word(w + 8 * i + 1, cb, rkg, c) << 32);
    const uint32_t rexp = (refill_word(ln < 4 ? 24 : 49, cb, rkg, c) >> (8 * (ln & 3))) & 0xffu;
    uint64_t z;
    const bool b = candidate<SIG, VAR>(cdt_sample<FULL>(v[1], v[0]), y[ln], v[2], rexp, kinv, z);
    cand[ln] = (uint32_t)z;
    bits = (bits & ~(0x101u << ln)) | candidate_bits(ln, b, z, k8);
  }
  return bits;
}

// Blocks of one refill that the fast path reads (16-byte block b = bytes 16b..16b+15, word w
// = bytes 4w..4w+3): 2, 3 (CDT words of lanes 0..3, words 8..15), 4, 5, 6 (Bernoulli words
// 16..24), 8..12 (CDT and Bernoulli words of lanes 4..7, words 33..49), 12..14 (the first 10
// uniform words from byte 200, words 50..59) and 17 (sign byte 280, word 70): 13 of the refill's
// 24 blocks.  Of each 64-bit CDT and Bernoulli word the fast path needs the top half only (the
// odd words of blocks 2..5, the even words of blocks 8..11), so 10 of the 13 blocks leave half of
// their final round out: 80 of the refill's 2,576 table lookups.  The low halves, and blocks 0,
// 1, 7 (the second CDT words, which only S3 uses), matter on ties; blocks 15 and 16 hold uniform
// words 60..67, needed only when fewer than 8 of the first 10 words are accepted.  The rare
// cases regenerate what they need on their slow paths.
//
// The blocks are computed in the order below and each is consumed as soon as it exists, so a
// refill never buffers its keystream: the sign byte, the uniform words and the CDT words first,
// then the Bernoulli words, two candidates at a time.  All live values (the 8 y, the packed CDT
// samples, a few words carried to a later block, the outputs) are registers; a buffered
// keystream had to live in local memory, whose traffic took 6% of the L1 data pipe that the
// table lookups saturate and missed L1 on a third of its loads.
//
// The order also keeps the recomputations of the counter cache (aes.cuh) rare.  The 32 refills of a
// warp start 24 counters apart from a multiple of 768, so in one lane the upper counter bits
// change between blocks 15 and 16, in one between blocks 7 and 8, and in no other inside the
// refill; a recomputation costs the whole warp 15 lookups.  Block 17 first and blocks 8..14 before
// blocks 2..6 makes 3 of them per refill (5 to 7 in other orders).
constexpr int kRefillBlocks = 13;
__constant__ uint8_t c_refill_order[kRefillBlocks] = {17, 12, 13, 14, 8, 9, 10, 11, 6, 2, 3, 4, 5};
// by step: bit s of kEvenWords / kOddWords -- words 0, 2 / words 1, 3 of that block are read
constexpr uint32_t kEvenWords = 0x01ffu;  // blocks 17, 12, 13, 14, 8..11 and 6
constexpr uint32_t kOddWords = 0x1e0eu;   // blocks 12, 13, 14 and 2..5

constexpr int kCandThreads = 512;  // 1 CTA (128 KiB of tables) per SM; 128 registers per thread

// Word W (0..9) of the branch-free uniform scan (src/gauss.c:578-703): the first 8 accepted
// words from byte 200 become y[0..7], kept in registers (the same 8 words in a shared-memory
// slot measured 17% slower on the whole kernel).  With at most 2 of the 10 words rejected
// (otherwise the slow path redoes the scan) word W lands in slot W - rej, rej = rejections
// before it, so only the slots W-2..W are candidates (3 selects per word, not 8); slots past
// 7 are dropped, as the reference's loop stops at 8 accepted words.
template <int SIG, int W>
__device__ __forceinline__ void uniform_step(uint32_t (&y)[8], uint32_t &rej, uint32_t be_word) {
  const uint32_t v = bswap32(be_word);
  const bool ok = uniform_ok<SIG>(v);
  const uint32_t r = uniform_reduce<SIG>(v);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (W - k >= 0 && W - k < 8) y[W - k] = (ok && rej == (uint32_t)k) ? r : y[W - k];
  rej += ok ? 0u : 1u;
}

template <int SIG, bool FULL, int VAR>
__global__ void __launch_bounds__(kCandThreads, 1)
    k_cand_cpu(const uint32_t *__restrict__ rkeys, SegDev sg, double kinv, uint32_t *__restrict__ cand_lo,
               uint8_t *__restrict__ amask, uint16_t *__restrict__ chs, uint32_t *__restrict__ status) {
  // the host keeps the flattened refill count below 2^32 - 2^24 (no wrap of g)
  const uint32_t total = (uint32_t)__ldg(sg.roff + sg.nstreams);
  // A contiguous run of refills per warp (the counter cache's upper part lasts 2,730 refills); warps are
  // dealt to the CTAs in turn, so that few refills spread over the SMs, where a warp alone is
  // three times as fast as one of 16.
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t run = ((total + warps - 1) / warps + 31u) & ~31u;
  if (blockIdx.x * run >= total) return;
  aes_fill_tables();
  __syncthreads();
  const AesCtx c = aes_ctx();
  uint32_t rk[60];
  uint32_t st = 0;
  uint32_t lo = 1, hi = 0;  // refill range of stream st (empty: forces the first lookup)
  CtrCache cc;
  const uint32_t g0 = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * run, g1 = min(total, g0 + run);
  for (uint32_t g = g0 + (threadIdx.x & 31u); g < g1; g += 32u) {
    if (g < lo || g >= hi) {
      st = seg_find(sg.roff, sg.nstreams, g);
      lo = (uint32_t)__ldg(sg.roff + st);
      hi = (uint32_t)__ldg(sg.roff + st + 1);
#pragma unroll
      for (int i = 0; i < 60; ++i) rk[i] = __ldg(rkeys + (size_t)st * 60 + i);
      ctr_cache_key(cc, rk, c);
    }
    const uint32_t *rkg = rkeys + (size_t)st * 60;  // the key schedule again, for rare paths
    const uint32_t t = g - lo;
    const uint32_t cb = t * 24u;
    uint32_t y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = 0;
    uint32_t rej = 0, k8 = 0, xp = 0, w34 = 0, w42 = 0, w48 = 0, ew = 0, lo0 = 0, lo1 = 0;
    uint32_t bits = 0;  // accept mask, bits 32 (<< 8), wide flag (bit 16)
    uint32_t open = 0;  // candidates that their top words do not decide
    uint32_t ln = 4;    // the next two candidates: ln, ln + 1 (lanes 4..7, then 0..3)
    // One AES body for all 13 blocks, one body for two CDT samples and one for two candidates
    // (src/gauss.c:836-890): the loop has to stay inside the instruction cache.  What is done with
    // a block is selected by the (warp-uniform) step.
#pragma unroll 1
    for (int step = 0; step < kRefillBlocks; ++step) {
      uint32_t W[4];
      aes256_ctr_block_cached(W, cb + c_refill_order[step], rk, rkg, c, cc, (kEvenWords >> step) & 1u,
                              (kOddWords >> step) & 1u);
      if (step == 0) {  // block 17: word 70 holds the sign byte 280
        k8 = bswap32(W[2]) & 0xffu;
      } else if (step == 1) {  // block 12: words 48 (top Bernoulli word of lane 7), 49 (exponents of lanes 4..7), 50, 51
        w48 = W[0];
        ew = W[1];
        uniform_step<SIG, 0>(y, rej, W[2]);
        uniform_step<SIG, 1>(y, rej, W[3]);
      } else if (step == 2) {  // block 13: uniform words 52..55
        uniform_step<SIG, 2>(y, rej, W[0]);
        uniform_step<SIG, 3>(y, rej, W[1]);
        uniform_step<SIG, 4>(y, rej, W[2]);
        uniform_step<SIG, 5>(y, rej, W[3]);
      } else if (step == 3) {  // block 14: uniform words 56..59; fewer than 8 of the 10 accepted: slow path
        uniform_step<SIG, 6>(y, rej, W[0]);
        uniform_step<SIG, 7>(y, rej, W[1]);
        uniform_step<SIG, 8>(y, rej, W[2]);
        uniform_step<SIG, 9>(y, rej, W[3]);
        if (rej > 2) {
          uint32_t ys[8];
          uniform_slow<SIG>(ys, 1, cb, rkg, c, status);
#pragma unroll
          for (int j = 0; j < 8; ++j) y[j] = ys[j];
        }
      } else if (step == 4) {  // block 8: top CDT word of lane 4 (34)
        w34 = W[2];
      } else if (step == 8) {  // block 6: word 24, the exponent bytes of lanes 0..3
        ew = W[0];
      } else if (step == 5 || step == 6 || step == 9 || step == 10) {
        // top CDT words, two lanes each: blocks 9 (lanes 5: 36, 6: 38), 10 (4: 34, 7: 40), 2 (0: 9, 1:
        // 11), 3 (2: 13, 3: 15); block 10 also has the top Bernoulli word of lane 4 (42).  xp holds the
        // samples of the next four candidates, 4 bits each.
        const uint32_t la = step == 5 ? 1u : step == 10 ? 2u : 0u, lb = step == 6 ? 3u : la + 1u;
        const uint32_t wa = step == 5 ? W[0] : step == 6 ? w34 : W[1];
        const uint32_t wb = step == 5 ? W[2] : step == 6 ? W[0] : W[3];
        if (step == 6) w42 = W[2];
        bool ta, tb;
        xp |= (cdt_sample_top(bswap32(wa), ta) << (4u * la)) | (cdt_sample_top(bswap32(wb), tb) << (4u * lb));
        open |= (((uint32_t)ta << la) | ((uint32_t)tb << lb)) << (step < 9 ? 4 : 0);
      } else {
        // top Bernoulli words: blocks 11 (lanes 4: 42, 5: 44 and 6: 46, 7: 48), 4 (0: 17, 1: 19), 5 (2:
        // 21, 3: 23).  Each pair of candidates takes its y, CDT samples and exponent bytes from the
        // head of their queues: y[4..7], y[0..3] in that order, xp and ew.
        uint32_t ra = step == 7 ? w42 : W[1], rb = step == 7 ? W[0] : W[3];
#pragma unroll 1
        for (;;) {
          uint64_t za, zb;
          bool ta, tb;
          const uint64_t va = candidate_input<SIG>(xp & 15u, y[4], za);
          const uint64_t vb = candidate_input<SIG>((xp >> 4) & 15u, y[5], zb);
          const bool ba = bernoulli_accept_top<SIG, VAR>(va, bswap32(ra), ew >> 24, kinv, ta);
          const bool bb = bernoulli_accept_top<SIG, VAR>(vb, bswap32(rb), (ew >> 16) & 0xffu, kinv, tb);
          bits |= candidate_bits(ln, ba, za, k8) | candidate_bits(ln + 1u, bb, zb, k8);
          open |= ((uint32_t)ta | ((uint32_t)tb << 1)) << ln;
          if (ln & 2u)
            reinterpret_cast<uint4 *>(cand_lo + (size_t)g * 8)[ln >> 2] = make_uint4(lo0, lo1, (uint32_t)za, (uint32_t)zb);
          lo0 = (uint32_t)za;
          lo1 = (uint32_t)zb;
          xp >>= 8;
          ew <<= 16;
          y[4] = y[6];
          y[5] = y[7];
          y[6] = y[0];
          y[7] = y[1];
          y[0] = y[2];
          y[1] = y[3];
          ln = (ln + 2u) & 7u;
          if (ln != 6u) break;
          ra = W[2];
          rb = w48;
        }
      }
    }
    if (open)
      bits = refill_slow<SIG, FULL, VAR>(open, k8, cb, rkg, c, kinv, cand_lo + (size_t)g * 8, bits, status);
    amask[g] = (uint8_t)bits;
    chs[g] = (uint16_t)(((bits >> 8) & 0xffu) | (k8 << 8));
    if (bits & 0x10000u) atomicOr(status, kStatusWideSample);
  }
}

// ------------------------------------------------------------------ CPU mapping, phase 2

constexpr int kScanTile = 4096;  // refills per scan tile (512 threads x 8)

// per-tile exclusive scan of accept counts: elocal[g] (within the tile), tile_sum[tile];
// one CTA per tile of the flattened tile space
__global__ void __launch_bounds__(512) k_scan_tiles(const uint8_t *__restrict__ amask, SegDev sg,
                                                    uint32_t *__restrict__ elocal, uint32_t *__restrict__ tile_sum) {
  __shared__ uint32_t wsum[16];
  const uint32_t T = blockIdx.x;
  const uint32_t st = seg_find(sg.toff, sg.nstreams, T);
  const uint64_t r0 = __ldg(sg.roff + st), R = __ldg(sg.roff + st + 1) - r0;
  const uint64_t base = (uint64_t)(T - __ldg(sg.toff + st)) * kScanTile + threadIdx.x * 8;
  uint32_t cnt[8], tot = 0;
  // whole runs at 8-byte aligned masks and 16-byte aligned prefixes (every refill range of a
  // uniform table in the 256-byte aligned scratch): one 8-byte load, two 16-byte stores
  const bool vec = base + 8 <= R && (reinterpret_cast<uintptr_t>(amask + r0 + base) & 7u) == 0 &&
                   (reinterpret_cast<uintptr_t>(elocal + r0 + base) & 15u) == 0;
  if (vec) {
    const uint2 m8 = __ldg(reinterpret_cast<const uint2 *>(amask + r0 + base));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      cnt[i] = __popc((m8.x >> (8 * i)) & 0xffu);
      cnt[4 + i] = __popc((m8.y >> (8 * i)) & 0xffu);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint64_t t = base + i;
      cnt[i] = t < R ? __popc(amask[r0 + t]) : 0u;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += cnt[i];
  // block exclusive scan of per-thread totals
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t s = lane < 16 ? wsum[lane] : 0u, si = s;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += v;
    }
    if (lane < 16) wsum[lane] = si - s;
    if (lane == 15) tile_sum[T] = si;
  }
  __syncthreads();
  uint32_t run = wsum[wid] + inc - tot;
  uint32_t ex[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    ex[i] = run;
    run += cnt[i];
  }
  if (vec) {
    uint4 *o = reinterpret_cast<uint4 *>(elocal + r0 + base);
    o[0] = make_uint4(ex[0], ex[1], ex[2], ex[3]);
    o[1] = make_uint4(ex[4], ex[5], ex[6], ex[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (base + i < R) elocal[r0 + base + i] = ex[i];
  }
}

// exclusive scan of the tile sums of each stream (one block per stream)
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t *__restrict__ tile_sum, SegDev sg) {
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t carry;
  const uint32_t st = blockIdx.x;
  const uint32_t t0 = __ldg(sg.toff + st), tiles = __ldg(sg.toff + st + 1) - t0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b0 = 0; b0 < tiles; b0 += 1024) {
    const uint32_t i = b0 + threadIdx.x;
    const uint32_t v = i < tiles ? tile_sum[t0 + i] : 0u;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
      uint32_t s = wsum[lane], si = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, si, o);
        if (lane >= o) si += u;
      }
      wsum[lane] = si - s;
    }
    __syncthreads();
    const uint32_t excl = carry + wsum[wid] + inc - v;
    if (i < tiles) tile_sum[t0 + i] = excl;
    __syncthreads();
    if (threadIdx.x == 1023) carry = excl + v;
    __syncthreads();
  }
}

// exclusive prefix E(t) of stream st's accept counts, t in [0, R]
struct SegView {
  uint64_t r0;
  uint32_t R, t0;
};
__device__ __forceinline__ SegView seg_view(const SegDev &sg, uint32_t st) {
  SegView v;
  v.r0 = __ldg(sg.roff + st);
  v.R = (uint32_t)(__ldg(sg.roff + st + 1) - v.r0);
  v.t0 = __ldg(sg.toff + st);
  return v;
}
__device__ __forceinline__ uint32_t prefix_at(const uint32_t *elocal, const uint32_t *tile_off, const uint8_t *amask,
                                              const SegView &v, uint32_t t) {
  if (t < v.R) return elocal[v.r0 + t] + tile_off[v.t0 + t / kScanTile];
  const uint32_t l = v.R - 1;
  return elocal[v.r0 + l] + tile_off[v.t0 + l / kScanTile] + __popc(amask[v.r0 + l]);
}

// one warp per stream: call c starts at a fresh refill a_c; it ends at the first refill e
// whose inclusive prefix reaches E(a_c) + n; a_{c+1} = e + 1.  call_start of stream st:
// coff[st] + st .. coff[st+1] + st (calls + 1 entries; the last is the end of the last call).
__global__ void k_walk(const uint32_t *__restrict__ elocal, const uint32_t *__restrict__ tile_off,
                       const uint8_t *__restrict__ amask, SegDev sg, float mean_accept,
                       uint32_t *__restrict__ call_start, uint32_t *__restrict__ status) {
  const uint32_t st = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (st >= sg.nstreams) return;  // whole warps only
  const SegView v = seg_view(sg, st);
  const uint32_t n = __ldg(sg.n + st), calls = __ldg(sg.calls + st);
  const uint32_t guess = (uint32_t)((float)n / mean_accept);
  uint32_t *cs = call_start + __ldg(sg.coff + st) + st;
  uint32_t a = 0;
  bool bad = v.R == 0;
  uint32_t c = 0;
  // exclusive prefix at a, the start of the current call; afterwards it is carried over from
  // the search, where the lane that found a call's last refill e has read prefix_at(e + 1)
  uint32_t base = bad ? 0u : prefix_at(elocal, tile_off, amask, v, 0);
  for (; c < calls && !bad; ++c) {
    const uint32_t target = base + n;
    // smallest e >= a whose inclusive prefix reaches target (monotone in e), searched in
    // windows of 32 refills around the expected call length; `known` is a position already
    // seen to satisfy (its prefix in known_pv).  Upward moves stop at the refill range,
    // downward moves at a.
    uint32_t lo = a + (guess > 16 ? guess - 16 : 0);
    int64_t known = -1;
    uint32_t known_pv = 0, e = 0, next_base = 0;
    for (int it = 0;; ++it) {
      if (it > (1 << 22)) {  // cannot happen for a monotone prefix; bounded regardless
        bad = true;
        break;
      }
      const uint32_t j = lo + lane;
      const uint32_t pv = j < v.R ? prefix_at(elocal, tile_off, amask, v, j + 1) : 0u;
      const bool ok = (j < v.R) && pv >= target;
      const uint32_t bal = __ballot_sync(0xffffffffu, ok);
      if (bal == 0) {
        if (known >= 0) {
          e = (uint32_t)known;
          next_base = known_pv;
          break;
        }
        if (lo + 32 >= v.R) {
          bad = true;
          break;
        }
        lo += 32;
        continue;
      }
      const int first = __ffs(bal) - 1;
      const uint32_t first_pv = __shfl_sync(0xffffffffu, pv, first);
      if (first > 0 || lo == a) {
        e = lo + first;
        next_base = first_pv;
        break;
      }
      known = lo;
      known_pv = first_pv;
      lo = lo > a + 32 ? lo - 32 : a;
    }
    if (bad) break;
    if (lane == 0) cs[c] = a;
    a = e + 1;
    base = next_base;
  }
  if (lane == 0) {
    if (bad) atomicOr(status, kStatusRefillsExhausted);
    for (uint32_t r = bad ? c : calls; r <= calls; ++r) cs[r] = bad ? v.R : a;
  }
}

// Pointer doubling for the call starts (the same result as k_walk).  next(t) of stream s is
// the refill after a call that starts at refill t ends: e + 1 for the first e >= t whose
// inclusive prefix reaches E(t) + n, or R + 1 (absorbing) when the stream runs out; the start
// of call c is next applied c times to 0, assembled from the bits of c with the tables
// J_k = next^(2^k).
__global__ void k_next_start(const uint32_t *__restrict__ elocal, const uint32_t *__restrict__ tile_off,
                             const uint8_t *__restrict__ amask, SegDev sg, float mean_accept,
                             uint32_t *__restrict__ next) {
  const uint64_t total = __ldg(sg.roff + sg.nstreams);
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const uint32_t st = seg_find(sg.roff, sg.nstreams, g);
  const SegView v = seg_view(sg, st);
  const uint32_t t = (uint32_t)(g - v.r0), n = __ldg(sg.n + st);
  const uint32_t target = prefix_at(elocal, tile_off, amask, v, t) + n;
  // smallest e in [t, R) with E(e + 1) >= target; try the expected call length first
  uint32_t lo = t, hi = v.R;
  const uint32_t guess = t + 2u * (uint32_t)((float)n / mean_accept) + 64u;
  if (guess < v.R && prefix_at(elocal, tile_off, amask, v, guess + 1) >= target) hi = guess;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (prefix_at(elocal, tile_off, amask, v, mid + 1) >= target) hi = mid;
    else lo = mid + 1;
  }
  next[g] = lo < v.R ? lo + 1 : v.R + 1;
}

__global__ void k_next_square(const uint32_t *__restrict__ jin, uint32_t *__restrict__ jout, SegDev sg) {
  const uint64_t total = __ldg(sg.roff + sg.nstreams);
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const uint32_t st = seg_find(sg.roff, sg.nstreams, g);
  const uint64_t r0 = __ldg(sg.roff + st);
  const uint32_t R = (uint32_t)(__ldg(sg.roff + st + 1) - r0);
  const uint32_t a = jin[g];
  jout[g] = a < R ? jin[r0 + a] : R + 1;
}

// one thread per (stream, c), c = 0 .. calls: call_start[coff[s] + s + c]
__global__ void k_starts_from_tables(const uint32_t *__restrict__ tables, int levels, uint64_t refills, SegDev sg,
                                     uint32_t *__restrict__ call_start, uint32_t *__restrict__ status) {
  const uint64_t total = __ldg(sg.coff + sg.nstreams) + sg.nstreams;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  uint32_t lo = 0, hi = sg.nstreams;  // stream s owns entries [coff[s] + s, coff[s+1] + s + 1)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(sg.coff + mid) + mid <= i) lo = mid;
    else hi = mid;
  }
  const uint32_t st = lo;
  const uint32_t c = (uint32_t)(i - (__ldg(sg.coff + st) + st));
  const uint64_t r0 = __ldg(sg.roff + st);
  const uint32_t R = (uint32_t)(__ldg(sg.roff + st + 1) - r0);
  uint32_t a = 0;
  for (int k = 0; k < levels; ++k)
    if ((c >> k) & 1u) a = a < R ? tables[(uint64_t)k * refills + r0 + a] : R + 1;
  call_start[i] = a <= R ? a : R;
  if (a > R && c == __ldg(sg.calls + st)) atomicOr(status, kStatusRefillsExhausted);
}

// ------------------------------------------------------------------ CPU mapping, phase 3

struct ModArgs {
  uint32_t q[3];
  uint64_t mu[3];   // floor(2^64 / q)
  uint32_t qr[3];   // floor(2^32 / q)
  uint32_t c32[3];  // 2^32 mod q
};

// (-1)^neg (hi 2^32 + lo) mod q_j for hi <= 1: lo mod q by one multiply-high (lo -
// floor(lo qr / 2^32) q is in [0, 2q)), plus 2^32 mod q when hi is set
__device__ __forceinline__ uint32_t residue_parts(uint32_t lo, uint32_t hi, uint32_t neg, const ModArgs &m, int j) {
  const uint32_t q = m.q[j];
  uint32_t r = mod_red1(lo - __umulhi(lo, m.qr[j]) * q, q);
  if (hi) r = mod_add(r, m.c32[j], q);
  return neg && r ? q - r : r;
}

// one CTA per call of the flattened call space: the accepted candidates of refills
// [a_c, a_{c+1}) in order, as residues out[ooff[st] + c * 3n ...][3][n].  Warp w of the CTA
// takes a contiguous run of the call's refills, 32 at a time: lane L loads the accept, bit-32
// and sign bits of refill t + L and, for k = 0..7, the low word of candidate L & 7 of refill
// t + 4k + L / 8 (eight coalesced 128-byte loads in flight per warp).  Per k the warp ballots the accepted lanes and packs
// them, in refill order and then candidate order (the order the reference consumes them), into
// a per-warp staging array; then every lane reduces one staged sample and the warp writes
// consecutive output positions.  Only the first position of each warp's run comes from the
// prefix tables.
constexpr int kScatterThreads = 256;
__global__ void __launch_bounds__(kScatterThreads)
    k_scatter(const uint32_t *__restrict__ cand_lo, const uint8_t *__restrict__ amask,
              const uint16_t *__restrict__ chs, const uint32_t *__restrict__ elocal,
              const uint32_t *__restrict__ tile_off, const uint32_t *__restrict__ call_start, SegDev sg, ModArgs m,
              uint32_t *__restrict__ out) {
  __shared__ uint2 stage[kScatterThreads / 32][256];
  const uint32_t st = seg_find(sg.coff, sg.nstreams, blockIdx.x);
  const uint64_t cs0 = __ldg(sg.coff + st);
  const uint32_t c = (uint32_t)(blockIdx.x - cs0);
  const SegView v = seg_view(sg, st);
  const uint32_t n = __ldg(sg.n + st);
  const uint32_t *cs = call_start + cs0 + st;
  const uint32_t a = cs[c], b = min(cs[c + 1], v.R);
  if (a >= b) return;
  const uint32_t lane = threadIdx.x & 31u, nw = blockDim.x >> 5;
  const uint32_t span = ((b - a + nw - 1) / nw + 3u) & ~3u;  // refills per warp
  const uint32_t t0 = a + (threadIdx.x >> 5) * span;
  if (t0 >= b) return;  // whole warps leave together; no CTA barrier follows
  const uint32_t t1 = min(t0 + span, b);
  uint32_t pos = prefix_at(elocal, tile_off, amask, v, t0) - prefix_at(elocal, tile_off, amask, v, a);
  uint32_t *o = out + __ldg(sg.ooff + st) + (size_t)c * 3 * n;
  uint2 *sw = stage[threadIdx.x >> 5];
  const uint32_t below = (1u << lane) - 1u, ci = lane & 7u;
  for (uint32_t t = t0; t < t1 && pos < n; t += 32) {
    // refill t + lane: accept bits, bit 32 of each |value| (<< 8), signs (<< 16)
    const uint32_t mk = t + lane < t1 ? (uint32_t)__ldg(amask + v.r0 + t + lane) |
                                            ((uint32_t)__ldg(chs + v.r0 + t + lane) << 8)
                                      : 0u;
    uint32_t lv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t r = t + 4 * k + (lane >> 3);
      lv[k] = r < t1 ? __ldg(cand_lo + (v.r0 + r) * 8 + ci) : 0u;
    }
    uint32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t meta = __shfl_sync(0xffffffffu, mk, 4 * k + (lane >> 3)) >> ci;
      const bool acc = meta & 1u;
      const uint32_t bal = __ballot_sync(0xffffffffu, acc);
      if (acc)  // staged as (low word, bit 32 | sign << 31)
        sw[cnt + __popc(bal & below)] = make_uint2(lv[k], ((meta >> 8) & 1u) | (((meta >> 16) & 1u) << 31));
      cnt += __popc(bal);
    }
    __syncwarp();
    for (uint32_t i = lane; i < cnt && pos + i < n; i += 32) {
      const uint2 sv = sw[i];
#pragma unroll
      for (int j = 0; j < 3; ++j) o[j * n + pos + i] = residue_parts(sv.x, sv.y & 1u, sv.y >> 31, m, j);
    }
    __syncwarp();  // the next step overwrites the staging array
    pos += cnt;
  }
}

// segment table of nstreams equal streams (calls x n each, refills R each, output stride
// `ostride` words per stream)
__global__ void k_seg_uniform(uint32_t nstreams, uint32_t calls, uint32_t n, uint32_t R, uint32_t tiles,
                              uint64_t ostride, uint32_t *__restrict__ sn, uint32_t *__restrict__ scalls,
                              uint64_t *__restrict__ roff, uint32_t *__restrict__ toff, uint64_t *__restrict__ coff,
                              uint64_t *__restrict__ ooff) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > nstreams) return;
  roff[i] = (uint64_t)i * R;
  toff[i] = i * tiles;
  coff[i] = (uint64_t)i * calls;
  if (i < nstreams) {
    sn[i] = n;
    scalls[i] = calls;
    ooff[i] = (uint64_t)i * ostride;
  }
}

// ------------------------------------------------------------------ GPU mapping

// The GPU mapping's refills are independent of each other: refill rep of thread t (n / 8 threads per
// polynomial, 8 samples each) starts at its own counter, poly * 5 T 24 + rep * T 24 + t 24 with
// T = n / 8, and chains its blocks (src/AES.cuh:380-435).  A task is one thread's 8 samples; it needs
// about 2.1 / 2.3 / 3.1 refills for S1 / S2 / S3.
struct ChainRefill {
  uint32_t z[8], y[8];  // low words of |candidate|; the uniform draws
  uint32_t bits;        // accept mask, bits 32 (<< 8), wide flag (bit 16); k8 << 24
};

// One refill from its full words, block by block (rare: a uniform draw beyond the first 10 words or a
// tied top word); the reference's order throughout.
template <int SIG>
__device__ __noinline__ void chain_refill_slow(uint32_t ctr, const uint32_t *__restrict__ rkg, AesCtx c, double kinv,
                                               ChainRefill &r, uint32_t *status) {
  uint32_t rk[60], buf[96];
#pragma unroll
  for (int i = 0; i < 60; ++i) rk[i] = __ldg(rkg + i);
  uint32_t s0 = rk[0], s1 = rk[1], s2 = rk[2], s3 = ctr ^ rk[3];
#pragma unroll 1
  for (int m = 0; m < 24; ++m) {
    aes256_rounds(s0, s1, s2, s3, rk, c);
    buf[4 * m] = s0, buf[4 * m + 1] = s1, buf[4 * m + 2] = s2, buf[4 * m + 3] = s3;
  }
  int w = 50;  // uniform words from byte 200
  const uint32_t k8 = buf[70] >> 24;  // byte 280
  r.bits = k8 << 24;
  for (int i = 0; i < 8; ++i) {
    uint32_t x = 0;
    for (;;) {
      if (w >= 96) {
        atomicOr(status, kStatusUniformOverrun);
        x = 0;
        break;
      }
      x = bswap32(buf[w++]);
      if (uniform_ok<SIG>(x)) break;
    }
    r.y[i] = uniform_reduce<SIG>(x);
  }
  for (int ln = 0; ln < 8; ++ln) {
    const int bw = (ln < 4 ? 0 : 25) + 2 * (ln & 3);
    const uint32_t x = cdt_sample<false>(le64_of(buf[bw + 8], buf[bw + 9]), 0);
    const uint32_t rexp = (buf[ln < 4 ? 24 : 49] >> (24 - 8 * (ln & 3))) & 0xffu;
    uint64_t z;
    const bool b = candidate<SIG, 2>(x, r.y[ln], le64_of(buf[bw + 16], buf[bw + 17]), rexp, kinv, z);
    r.z[ln] = (uint32_t)z;
    r.bits |= candidate_bits(ln, b, z, k8);
  }
}

// A warp runs a contiguous range of tasks, `group` lanes (1 or 4) per task: with 1, a lane that has its
// 8 samples takes the warp's next task at once, so no lane waits for the slowest of 32; with 4 the
// lanes draw consecutive refills of one task, the shortest way through a call with few tasks.
// Warps are dealt to the CTAs in turn, so that few warps spread over the SMs.
//
// A refill's 18 blocks are a serial chain, so they come in order and what needs a later word waits in
// registers: CDT samples and top Bernoulli words until the uniform draws (blocks 12..14), the
// candidates until the sign byte (block 17).  Top words decide as in the CPU mapping (k_cand_cpu).
// Bound by the table lookups: 4,020 per refill, 16 cycles of a warp's round against 12 of the ALU.
// One CTA of 512 tasks with its own tables, a buffered keystream and lanes that waited for the slowest
// of their warp took 901 us for 785 polynomials of S3 and 159 for one of S2 on a B200 (n = 4096); now 525 and 20.
constexpr int kGpuMapThreads = 512;
template <int SIG>
__global__ void __launch_bounds__(kGpuMapThreads, 1)
    k_gauss_gpu_map(const uint32_t *__restrict__ rkey, uint32_t poly0, uint32_t tasks, uint32_t n, uint32_t run,
                    uint32_t group, double kinv, ModArgs m, uint32_t *__restrict__ out, uint32_t *__restrict__ status) {
  const uint32_t T = n / 8, lane = threadIdx.x & 31u;
  if ((uint64_t)blockIdx.x * run >= tasks) return;  // no task for this CTA's first warp, nor for the others
  aes_fill_tables();
  __syncthreads();
  const uint32_t wi = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint64_t first = (uint64_t)wi * run;
  if (first >= tasks) return;
  const uint32_t end = (uint32_t)min((uint64_t)tasks, first + run);
  uint32_t next = (uint32_t)first;
  const AesCtx c = aes_ctx();
  uint32_t rk[60];
#pragma unroll
  for (int i = 0; i < 60; ++i) rk[i] = __ldg(rkey + i);
  const uint32_t leader = lane & ~(group - 1u), rank = lane & (group - 1u);
  uint32_t task = 0xffffffffu, rep = 0, have = 0;  // the lane's task, the refills and samples it has
  for (;;) {
    // lanes without a task take the next ones of the warp's range
    const uint32_t idle = __ballot_sync(0xffffffffu, task == 0xffffffffu && rank == 0);
    if (task == 0xffffffffu) {
      const uint32_t at = next + __popc(idle & ((1u << leader) - 1u));
      if (at < end) task = at, rep = 0, have = 0;
    }
    next += __popc(idle);
    const bool live = task != 0xffffffffu;
    if (!__any_sync(0xffffffffu, live)) break;
    const uint32_t p = live ? task / T : 0u, t = live ? task - p * T : 0u;
    const uint32_t ctr = (poly0 + p) * 5u * T * 24u + (rep + rank) * T * 24u + t * 24u;
    uint32_t s0 = rk[0], s1 = rk[1], s2 = rk[2], s3 = ctr ^ rk[3];
    uint32_t y[8], rm[8], zl[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = 0;
    uint32_t rej = 0, xp = 0, e0 = 0, e1 = 0, w34 = 0, bits = 0, open = 0, k8 = 0;
#pragma unroll 1
    for (int blk = 0; blk < 18; ++blk) {
      aes256_rounds(s0, s1, s2, s3, rk, c);
      if (blk == 2 || blk == 3 || blk == 9 || blk == 10) {  // top CDT words of two lanes
        const uint32_t la = blk == 2 ? 0u : blk == 3 ? 2u : blk == 9 ? 5u : 4u, lb = blk == 10 ? 7u : la + 1u;
        const uint32_t wa = blk < 4 ? s1 : blk == 9 ? s0 : w34, wb = blk < 4 ? s3 : blk == 9 ? s2 : s0;
        bool ta, tb;
        xp |= (cdt_sample_top(bswap32(wa), ta) << (4u * la)) | (cdt_sample_top(bswap32(wb), tb) << (4u * lb));
        open |= (uint32_t)(ta | tb);
        if (blk == 10) rm[4] = s2;
      } else if (blk == 4) {
        rm[0] = s1, rm[1] = s3;
      } else if (blk == 5) {
        rm[2] = s1, rm[3] = s3;
      } else if (blk == 6) {
        e0 = s0;
      } else if (blk == 8) {
        w34 = s2;
      } else if (blk == 11) {
        rm[5] = s0, rm[6] = s2;
      } else if (blk == 12) {
        rm[7] = s0, e1 = s1;
        uniform_step<SIG, 0>(y, rej, s2);
        uniform_step<SIG, 1>(y, rej, s3);
      } else if (blk == 13) {
        uniform_step<SIG, 2>(y, rej, s0);
        uniform_step<SIG, 3>(y, rej, s1);
        uniform_step<SIG, 4>(y, rej, s2);
        uniform_step<SIG, 5>(y, rej, s3);
      } else if (blk == 14) {
        uniform_step<SIG, 6>(y, rej, s0);
        uniform_step<SIG, 7>(y, rej, s1);
        uniform_step<SIG, 8>(y, rej, s2);
        uniform_step<SIG, 9>(y, rej, s3);
      } else if (blk == 17) {
        k8 = s2 >> 24;  // byte 280
      }
    }
    // the candidates, two at a time through one body
#pragma unroll 1
    for (uint32_t ln = 0; ln < 8; ln += 2) {
      uint64_t za, zb;
      bool ta, tb;
      const uint64_t va = candidate_input<SIG>(xp & 15u, y[0], za);
      const uint64_t vb = candidate_input<SIG>((xp >> 4) & 15u, y[1], zb);
      const bool ba = bernoulli_accept_top<SIG, 2>(va, bswap32(rm[0]), e0 >> 24, kinv, ta);
      const bool bb = bernoulli_accept_top<SIG, 2>(vb, bswap32(rm[1]), (e0 >> 16) & 0xffu, kinv, tb);
      bits |= candidate_bits((int)ln, ba, za, k8) | candidate_bits((int)ln + 1, bb, zb, k8);
      open |= (uint32_t)(ta | tb);
#pragma unroll
      for (int i = 0; i < 6; ++i) y[i] = y[i + 2], rm[i] = rm[i + 2], zl[i] = zl[i + 2];
      zl[6] = (uint32_t)za;
      zl[7] = (uint32_t)zb;
      xp >>= 8;
      e0 = ln == 2 ? e1 : e0 << 16;
    }
    if (live && (open | (uint32_t)(rej > 2))) {
      ChainRefill r;
      chain_refill_slow<SIG>(ctr, rkey, c, kinv, r, status);
      bits = r.bits & 0x00ffffffu;
      k8 = r.bits >> 24;
#pragma unroll
      for (int i = 0; i < 8; ++i) zl[i] = r.z[i];
    }
    if (live && (bits & 0x10000u)) atomicOr(status, kStatusWideSample);
    // positions: the samples of this task's earlier lanes come first
    uint32_t cnt = live ? __popc(bits & 0xffu) : 0u, pos = have, total = cnt;
    for (uint32_t d = 1; d < group; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, total, d);
      if (rank >= d) total += o;
    }
    pos += total - cnt;
    have += __shfl_sync(0xffffffffu, total, leader + group - 1u);
    if (live) {
      uint32_t *o = out + (size_t)p * 3 * n + 8 * t;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (((bits >> i) & 1u) && pos < 8) {
#pragma unroll
          for (int j = 0; j < 3; ++j)
            o[j * n + pos] = residue_parts(zl[i], (bits >> (8 + i)) & 1u, (k8 >> i) & 1u, m, j);
          ++pos;
        }
      }
      rep += group;
      if (have >= 8) {
        task = 0xffffffffu;
      } else if (rep >= kMaxRefillsPerThread) {  // never reached by a working sampler; bounded anyway
        atomicOr(status, kStatusRefillCap);
        task = 0xffffffffu;
      }
    }
  }
}

// ------------------------------------------------------------------ uniform a

// sample_polya (src/sample.c:56-128): AES-CTR (nonce 0) bytes, a_i = le64(bytes 8i..8i+7) mod q_j
__global__ void __launch_bounds__(256) k_polya(const uint32_t *__restrict__ rkey, uint32_t n, ModArgs m,
                                               uint32_t *__restrict__ a) {
  aes_fill_tables();
  __syncthreads();
  const AesCtx c = aes_ctx();
  uint32_t rk[60];
#pragma unroll
  for (int i = 0; i < 60; ++i) rk[i] = __ldg(rkey + i);
  const uint32_t blk = blockIdx.x * blockDim.x + threadIdx.x;
  if (blk >= n / 2) return;
  uint32_t W[4];
  aes256_ctr_block(W, 0u, blk, rk, c);
  const uint64_t v0 = le64_of(W[0], W[1]), v1 = le64_of(W[2], W[3]);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    a[j * n + 2 * blk] = mod_u64(v0, m.mu[j], m.q[j]);
    a[j * n + 2 * blk + 1] = mod_u64(v1, m.mu[j], m.q[j]);
  }
}

}  // namespace

// ------------------------------------------------------------------ host side


static ModArgs mod_args() {
  ModArgs m;
  for (int j = 0; j < 3; ++j) {
    m.q[j] = kRefPrimes[j];
    unsigned __int128 one = (unsigned __int128)1 << 64;
    m.mu[j] = (uint64_t)(one / kRefPrimes[j]);
    m.qr[j] = (uint32_t)((1ull << 32) / kRefPrimes[j]);
    m.c32[j] = (uint32_t)((1ull << 32) % kRefPrimes[j]);
  }
  return m;
}

static double kinv_of(int sig) {
  const uint64_t K = sigma_k(sig);
  return -1.0 / (double)(int64_t)(K * K);
}

static uint8_t gmul8(uint8_t a, uint8_t b) {
  uint8_t r = 0;
  while (b) {
    if (b & 1) r ^= a;
    a = (uint8_t)((a << 1) ^ ((a & 0x80) ? 0x1b : 0));
    b >>= 1;
  }
  return r;
}

void aes_key_expand(const uint8_t key[32], uint32_t w[60]) {
  static uint8_t sbox[256];
  static bool ready = false;
  if (!ready) aes_sbox(sbox), ready = true;
  uint8_t rc = 1;
  for (int i = 0; i < 8; ++i)
    w[i] = ((uint32_t)key[4 * i] << 24) | ((uint32_t)key[4 * i + 1] << 16) | ((uint32_t)key[4 * i + 2] << 8) |
           key[4 * i + 3];
  for (int i = 8; i < 60; ++i) {
    uint32_t t = w[i - 1];
    auto sub = [&](uint32_t v) {
      return ((uint32_t)sbox[v >> 24] << 24) | ((uint32_t)sbox[(v >> 16) & 255] << 16) |
             ((uint32_t)sbox[(v >> 8) & 255] << 8) | sbox[v & 255];
    };
    if (i % 8 == 0) {
      t = sub((t << 8) | (t >> 24)) ^ ((uint32_t)rc << 24);
      rc = gmul8(rc, 2);
    } else if (i % 8 == 4) {
      t = sub(t);
    }
    w[i] = w[i - 8] ^ t;
  }
}

void aes_sbox(uint8_t out[256]) {
  // FIPS-197 5.1.1: multiplicative inverse in GF(2^8) followed by the affine map
  for (int x = 0; x < 256; ++x) {
    uint8_t inv = 0;
    if (x)
      for (int y = 1; y < 256; ++y)
        if (gmul8((uint8_t)x, (uint8_t)y) == 1) {
          inv = (uint8_t)y;
          break;
        }
    uint8_t s = inv;
    for (int r = 1; r <= 4; ++r) s ^= (uint8_t)((inv << r) | (inv >> (8 - r)));
    out[x] = s ^ 0x63;
  }
}

// AES-256 key expansion (FIPS-197 5.2) on the device, one key per thread, into the
// big-endian round-key words of aes_key_expand: rk[i][60] from seeds[perm ? perm[i] : i][32]
__global__ void k_expand_keys(const uint8_t *__restrict__ seeds, const uint32_t *__restrict__ perm, uint32_t count,
                              uint32_t *__restrict__ rk) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint8_t *k = seeds + 32 * (size_t)(perm ? perm[i] : i);
  uint32_t w[60];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    w[j] = ((uint32_t)k[4 * j] << 24) | ((uint32_t)k[4 * j + 1] << 16) | ((uint32_t)k[4 * j + 2] << 8) | k[4 * j + 3];
#pragma unroll
  for (int j = 8; j < 60; ++j) {
    uint32_t t = w[j - 1];
    if (j % 8 == 0) t = (t << 8) | (t >> 24);
    if (j % 8 == 0 || j % 8 == 4)
      t = ((uint32_t)c_sbox[t >> 24] << 24) | ((uint32_t)c_sbox[(t >> 16) & 255] << 16) |
          ((uint32_t)c_sbox[(t >> 8) & 255] << 8) | c_sbox[t & 255];
    if (j % 8 == 0) t ^= (1u << (j / 8 - 1)) << 24;  // round constants 1, 2, 4, ..., 64
    w[j] = w[j - 8] ^ t;
  }
  uint32_t *o = rk + (size_t)i * 60;
#pragma unroll
  for (int j = 0; j < 60; ++j) o[j] = w[j];
}

int expand_keys_device(const uint8_t *d_seeds, const uint32_t *d_perm, uint32_t count, uint32_t *d_rk,
                       cudaStream_t s) {
  if (!count) return CUFE_OK;
  note_launch(), k_expand_keys<<<(count + 127) / 128, 128, 0, s>>>(d_seeds, d_perm, count, d_rk);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

int sampler_init_device() {
  uint8_t sbox[256];
  aes_sbox(sbox);
  CUFE_CUDA(cudaMemcpyToSymbol(c_sbox, sbox, 256));
  CUFE_CUDA(cudaFuncSetAttribute(k_cand_cpu<0, false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_cand_cpu<1, false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_cand_cpu<2, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_gauss_gpu_map<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_gauss_gpu_map<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_gauss_gpu_map<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  CUFE_CUDA(cudaFuncSetAttribute(k_polya, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes));
  return CUFE_OK;
}

// Accepted candidates per 8-candidate refill of the CPU mapping, measured on the oracle over
// 4 M AES-CTR refills per sigma: mean 5.4436 / 4.3942 / 3.0948 (+-0.0007) and variance 1.74 /
// 1.98 / 1.90 for S1 / S2 / S3 (the uint32 truncation of src/gauss.c:849 rejects more at large
// K).  The means below are those rounded down, the variance bound is 2.0 for all three.
static double mean_accept(int sig) { return sig == 0 ? 5.443 : (sig == 1 ? 4.393 : 3.094); }
constexpr double kAcceptVarBound = 2.0;

// Refills precomputed for `calls` consecutive calls of n samples.  A call consumes r refills,
// the first whose accepted total reaches n; E[r] = (n + overshoot) / mu < n / mu + 1 (the
// overshoot averages below 1.4 samples), and over many calls sum(r) has variance about
// calls n v / mu^3 (renewal count).  The range is calls (n / mu + 1) plus 12 of those
// standard deviations plus 64.  Against the exact distribution of r (dynamic programming
// over the measured accept-count histogram), that is at least 13 standard deviations of
// sum(r) above its mean for every n in 16..8192 and 1..4096 calls, and 0.2-0.6% above the
// mean need for long streams (the former 3% margin over rounded-down means was 6%).  A
// stream that still ran short sets kStatusRefillsExhausted (checked by the host) and never
// reads past its range.
uint32_t cpu_map_refills(uint32_t calls, uint32_t n, int sig) {
  const double mu = mean_accept(sig), cn = (double)calls * (double)n;
  const double need = (double)calls * ((double)n / mu + 1.0);
  const double sd = std::sqrt(cn * kAcceptVarBound / (mu * mu * mu));
  const uint32_t R = (uint32_t)std::ceil(need + 12.0 * sd) + 64;
  return (R + 31) & ~31u;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

SegLayout seg_layout(uint32_t S) {
  SegLayout L;
  size_t o = 0;
  L.n = o;
  o += align256((size_t)S * 4);
  L.calls = o;
  o += align256((size_t)S * 4);
  L.toff = o;
  o += align256((size_t)(S + 1) * 4);
  L.roff = o;
  o += align256((size_t)(S + 1) * 8);
  L.coff = o;
  o += align256((size_t)(S + 1) * 8);
  L.ooff = o;
  o += align256((size_t)S * 8);
  L.bytes = o;
  return L;
}

SegDev seg_bind(void *base, uint32_t S) {
  const SegLayout L = seg_layout(S);
  uint8_t *b = static_cast<uint8_t *>(base);
  SegDev d;
  d.nstreams = S;
  d.n = reinterpret_cast<const uint32_t *>(b + L.n);
  d.calls = reinterpret_cast<const uint32_t *>(b + L.calls);
  d.toff = reinterpret_cast<const uint32_t *>(b + L.toff);
  d.roff = reinterpret_cast<const uint64_t *>(b + L.roff);
  d.coff = reinterpret_cast<const uint64_t *>(b + L.coff);
  d.ooff = reinterpret_cast<const uint64_t *>(b + L.ooff);
  return d;
}

SegSizes seg_fill_host(int sig, uint32_t S, const uint32_t *calls, const uint32_t *n, const uint64_t *ooff,
                       void *host_base) {
  const SegLayout L = seg_layout(S);
  uint8_t *b = static_cast<uint8_t *>(host_base);
  uint32_t *hn = reinterpret_cast<uint32_t *>(b + L.n), *hc = reinterpret_cast<uint32_t *>(b + L.calls);
  uint32_t *ht = reinterpret_cast<uint32_t *>(b + L.toff);
  uint64_t *hr = reinterpret_cast<uint64_t *>(b + L.roff), *hco = reinterpret_cast<uint64_t *>(b + L.coff);
  uint64_t *ho = reinterpret_cast<uint64_t *>(b + L.ooff);
  SegSizes z{S, 0, 0, 0, 0, false};
  for (uint32_t i = 0; i < S; ++i) {
    const uint32_t R = cpu_map_refills(calls[i], n[i], sig);
    hn[i] = n[i];
    hc[i] = calls[i];
    ho[i] = ooff ? ooff[i] : 0;
    hr[i] = z.refills;
    ht[i] = z.tiles;
    hco[i] = z.calls;
    z.refills += R;
    z.tiles += (R + kScanTile - 1) / kScanTile;
    z.calls += calls[i];
    z.max_calls = std::max(z.max_calls, calls[i]);
  }
  hr[S] = z.refills;
  ht[S] = z.tiles;
  hco[S] = z.calls;
  z.doubling = seg_auto_doubling(z.refills, z.max_calls);
  return z;
}

static SegSizes seg_uniform_sizes(uint32_t S, uint32_t calls, uint32_t n, int sig) {
  const uint32_t R = cpu_map_refills(calls, n, sig);
  return SegSizes{S, (uint64_t)S * R, S * ((R + kScanTile - 1) / kScanTile), (uint64_t)S * calls, calls,
                  seg_auto_doubling((uint64_t)S * R, calls)};
}

static int g_call_search = 0;
void set_call_search(int mode) { g_call_search = mode; }
int get_call_search() { return g_call_search; }

constexpr uint64_t kDoublingMaxRefills = (uint64_t)32 << 20;

static int doubling_levels(uint32_t max_calls) {
  int k = 1;
  while (k < 31 && (1u << k) <= max_calls) ++k;
  return k;  // bit_length(max_calls), at least 1
}
// Doubling costs about 6.4 ps per refill per table level (memory-bound gathers); the walk
// about 1.0-1.4 us per call of its longest stream (serial dependent loads), both measured on
// a B200 (sigma_3 at n = 4096, l = 784: doubling 0.48 / 1.12 ms at 8 / 16 encryptions, walk
// 0.78 ms up to 16 and 1.13 ms from 24).  Doubling is chosen when it is the cheaper of the two
// and its tables stay below 32 Mi refills.
bool seg_auto_doubling(uint64_t refills, uint32_t max_calls) {
  if (g_call_search == 1 || refills > kDoublingMaxRefills) return false;
  if (g_call_search == 2) return true;
  return refills * (uint64_t)doubling_levels(max_calls) <= (uint64_t)max_calls * 200000u;
}

size_t seg_scratch_bytes(const SegSizes &z) {
  size_t b = align256(z.refills * 32) + align256(z.refills) + align256(z.refills * 2) + align256(z.refills * 4) +
             align256((size_t)z.tiles * 4) +
             align256((z.calls + z.nstreams) * 4);
  if (z.doubling) b += (size_t)doubling_levels(z.max_calls) * align256(z.refills * 4);
  return b;
}

size_t cpu_map_workspace_bytes(uint32_t nstreams, uint32_t calls, uint32_t n, int sig) {
  return seg_layout(nstreams).bytes + seg_scratch_bytes(seg_uniform_sizes(nstreams, calls, n, sig));
}

int sample_cpu_map_seg(int sig, const SegDev &sg, const SegSizes &z, const uint32_t *d_rkeys, uint32_t *d_out,
                       void *scratch, uint32_t *d_status, int num_sms, cudaStream_t s) {
  if (sig < 0 || sig > 2 || z.nstreams == 0 || z.tiles >= (1u << 31) || z.calls >= (1ull << 31) ||
      z.refills >= (1ull << 32) - (1ull << 24))
    return CUFE_ERR_INVALID;
  uint8_t *p = static_cast<uint8_t *>(scratch);
  auto take = [&](size_t x) {
    uint8_t *r = p;
    p += align256(x);
    return r;
  };
  uint32_t *cand = reinterpret_cast<uint32_t *>(take(z.refills * 32));  // low words of |candidate|
  uint8_t *amask = take(z.refills);
  uint16_t *chs = reinterpret_cast<uint16_t *>(take(z.refills * 2));  // bit 32 of each, signs << 8
  uint32_t *elocal = reinterpret_cast<uint32_t *>(take(z.refills * 4));
  uint32_t *tsum = reinterpret_cast<uint32_t *>(take((size_t)z.tiles * 4));
  uint32_t *cstart = reinterpret_cast<uint32_t *>(take((z.calls + z.nstreams) * 4));
  const double kinv = kinv_of(sig);
  const uint32_t grid =
      (uint32_t)std::min<uint64_t>((uint64_t)num_sms, (z.refills + 31) / 32);
  if (grid > 0) {
    ProfScope ps(sig == 0 ? "sample_cand_s1" : (sig == 1 ? "sample_cand_s2" : "sample_cand_s3"), s);
    if (sig == 0)
      note_launch(), k_cand_cpu<0, false, 0><<<grid, kCandThreads, kAesSmemBytes, s>>>(d_rkeys, sg, kinv, cand, amask, chs,
                                                                             d_status);
    else if (sig == 1)
      note_launch(), k_cand_cpu<1, false, 0><<<grid, kCandThreads, kAesSmemBytes, s>>>(d_rkeys, sg, kinv, cand, amask, chs,
                                                                             d_status);
    else
      note_launch(), k_cand_cpu<2, true, 1><<<grid, kCandThreads, kAesSmemBytes, s>>>(d_rkeys, sg, kinv, cand, amask, chs,
                                                                             d_status);
  }
  CUFE_CUDA(cudaGetLastError());
  if (z.tiles) {
    ProfScope ps("sample_scan", s);
    note_launch(), k_scan_tiles<<<z.tiles, 512, 0, s>>>(amask, sg, elocal, tsum);
    note_launch(), k_scan_sums<<<z.nstreams, 1024, 0, s>>>(tsum, sg);
  }
  if (z.doubling) {
    const int levels = doubling_levels(z.max_calls);
    uint32_t *tab = reinterpret_cast<uint32_t *>(take((size_t)levels * align256(z.refills * 4)));
    const uint64_t stride = align256(z.refills * 4) / 4;
    ProfScope ps("sample_walk", s);
    const unsigned rg = (unsigned)((z.refills + 255) / 256);
    note_launch(), k_next_start<<<rg, 256, 0, s>>>(elocal, tsum, amask, sg, (float)mean_accept(sig), tab);
    for (int k = 1; k < levels; ++k) note_launch(), k_next_square<<<rg, 256, 0, s>>>(tab + (k - 1) * stride, tab + k * stride, sg);
    note_launch(), k_starts_from_tables<<<(unsigned)((z.calls + z.nstreams + 255) / 256), 256, 0, s>>>(tab, levels, stride, sg,
                                                                                        cstart, d_status);
  } else {
    ProfScope ps("sample_walk", s);
    note_launch(), k_walk<<<(z.nstreams + 3) / 4, 128, 0, s>>>(elocal, tsum, amask, sg, (float)mean_accept(sig), cstart, d_status);
  }
  CUFE_CUDA(cudaGetLastError());
  if (d_out && z.calls) {
    ProfScope ps_sc("sample_scatter", s);
    note_launch(), k_scatter<<<(uint32_t)z.calls, kScatterThreads, 0, s>>>(cand, amask, chs, elocal, tsum, cstart, sg,
                                                                           mod_args(), d_out);
    CUFE_CUDA(cudaGetLastError());
  }
  return CUFE_OK;
}

// the uniform case: nstreams equal streams, tables built on the device (capturable)
static int seg_uniform(uint32_t nstreams, uint32_t calls, uint32_t n, int sig, void *ws, cudaStream_t s, SegDev *sg,
                       SegSizes *z, void **scratch) {
  const SegLayout L = seg_layout(nstreams);
  *z = seg_uniform_sizes(nstreams, calls, n, sig);
  if (z->refills / nstreams >= (1ull << 32) / 24) return CUFE_ERR_INVALID;  // AES counter range
  uint8_t *b = static_cast<uint8_t *>(ws);
  *sg = seg_bind(b, nstreams);
  const uint32_t R = (uint32_t)(z->refills / nstreams);
  note_launch(), k_seg_uniform<<<(nstreams + 256) / 256, 256, 0, s>>>(
      nstreams, calls, n, R, z->tiles / nstreams, (uint64_t)calls * 3 * n, reinterpret_cast<uint32_t *>(b + L.n),
      reinterpret_cast<uint32_t *>(b + L.calls), reinterpret_cast<uint64_t *>(b + L.roff),
      reinterpret_cast<uint32_t *>(b + L.toff), reinterpret_cast<uint64_t *>(b + L.coff),
      reinterpret_cast<uint64_t *>(b + L.ooff));
  CUFE_CUDA(cudaGetLastError());
  *scratch = b + L.bytes;
  return CUFE_OK;
}

int sample_cpu_map(int sig, uint32_t nstreams, const uint32_t *d_rkeys, uint32_t calls, uint32_t n,
                   uint32_t *d_out, void *ws, uint32_t *d_status, int num_sms, cudaStream_t s) {
  SegDev sg;
  SegSizes z;
  void *scratch;
  int rc = seg_uniform(nstreams, calls, n, sig, ws, s, &sg, &z, &scratch);
  if (rc) return rc;
  return sample_cpu_map_seg(sig, sg, z, d_rkeys, d_out, scratch, d_status, num_sms, s);
}

int sample_gpu_map(int sig, const uint32_t *d_rkey, uint32_t poly0, uint32_t npolys, uint32_t n, uint32_t *d_out,
                   uint32_t *d_status, int num_sms, cudaStream_t s) {
  const uint32_t tasks = npolys * (n / 8);
  const uint32_t warps = (uint32_t)num_sms * (kGpuMapThreads / 32);
  // 4 lanes per task while that leaves at most half of the warps a task group
  const uint32_t group = (uint64_t)tasks * 4 <= (uint64_t)warps * 16 ? 4u : 1u;
  const uint32_t run = std::max((tasks + warps - 1) / warps, 32u / group);
  const uint32_t grid = std::min<uint32_t>((uint32_t)num_sms, (tasks + run - 1) / run);
  const double kinv = kinv_of(sig);
  ProfScope ps("sample_gpu_map", s);
  note_launch();
  if (sig == 0)
    k_gauss_gpu_map<0><<<grid, kGpuMapThreads, kAesSmemBytes, s>>>(d_rkey, poly0, tasks, n, run, group, kinv, mod_args(),
                                                                   d_out, d_status);
  else if (sig == 1)
    k_gauss_gpu_map<1><<<grid, kGpuMapThreads, kAesSmemBytes, s>>>(d_rkey, poly0, tasks, n, run, group, kinv, mod_args(),
                                                                   d_out, d_status);
  else
    k_gauss_gpu_map<2><<<grid, kGpuMapThreads, kAesSmemBytes, s>>>(d_rkey, poly0, tasks, n, run, group, kinv, mod_args(),
                                                                   d_out, d_status);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

int sample_polya(const uint32_t *d_rkey, uint32_t n, uint32_t *d_a, cudaStream_t s) {
  const uint32_t grid = (n / 2 + 255) / 256;
  ProfScope ps("sample_polya", s);
  note_launch(), k_polya<<<grid, 256, kAesSmemBytes, s>>>(d_rkey, n, mod_args(), d_a);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

}  // namespace cufe

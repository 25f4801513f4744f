// sampler.cu -- AES-256-CTR keystreams and the discrete Gaussian / uniform samplers.
//
// Two counter-to-sample mappings are implemented, both bit-exact:
//
//  * CPU mapping (src/gauss.c + src/aes256ctr.c): one AES-CTR stream per context; every
//    gaussian_sampler_* call consumes 384-byte refills (24 counter blocks) in order, takes
//    the accepted candidates in order and drops the rest of its last refill.  The stream is
//    sequential by construction, so it is computed in three parallel phases: (1) every
//    refill's 8 candidates and accept mask for a generous refill range (the AES work, one
//    thread per refill), (2) a search per stream over the accept counts that finds where each
//    call starts (each call starts at a fresh refill), (3) a
//    scatter of the accepted candidates to their coefficient positions as residues.
//  * GPU mapping (src/sample_gpu.cu, src/AES.cuh): thread t of polynomial p owns coefficients
//    8t..8t+7 and draws chained-AES refills from counter p*5*T*24 + rep*T*24 + t*24.
#include "aes.cuh"
#include "sampler.cuh"
#include "sampler_host.h"
#include "scheme.cuh"
#include "prof.h"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace cufe {

namespace {

__device__ __forceinline__ uint64_t le64_of(uint32_t be_lo, uint32_t be_hi) {
  return (uint64_t)bswap32(be_lo) | ((uint64_t)bswap32(be_hi) << 32);
}

// ------------------------------------------------------------------ segment tables

// The tables of a run with different streams, or the arithmetic of one with equal streams
__device__ __forceinline__ uint32_t seg_n(const SegDev &sg, uint32_t st) { return sg.n ? __ldg(sg.n + st) : sg.u_n; }
__device__ __forceinline__ uint32_t seg_calls(const SegDev &sg, uint32_t st) {
  return sg.n ? __ldg(sg.calls + st) : sg.u_calls;
}
__device__ __forceinline__ uint64_t seg_roff(const SegDev &sg, uint32_t st) {
  return sg.n ? __ldg(sg.roff + st) : (uint64_t)st * sg.u_refills;
}
__device__ __forceinline__ uint64_t seg_coff(const SegDev &sg, uint32_t st) {
  return sg.n ? __ldg(sg.coff + st) : (uint64_t)st * sg.u_calls;
}
__device__ __forceinline__ uint64_t seg_ooff(const SegDev &sg, uint32_t st) {
  return sg.n ? __ldg(sg.ooff + st) : st * sg.u_ostride;
}
__device__ __forceinline__ uint32_t seg_of_refill(const SegDev &sg, uint32_t g) {
  return sg.n ? seg_find(sg.roff, sg.nstreams, g) : g / sg.u_refills;
}
__device__ __forceinline__ uint32_t seg_of_call(const SegDev &sg, uint32_t c) {
  return sg.n ? seg_find(sg.coff, sg.nstreams, c) : c / sg.u_calls;
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

// kCandThreads = 512: 1 CTA (192 KiB of tables) per SM; 128 registers per thread

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
  const uint32_t total = (uint32_t)seg_roff(sg, sg.nstreams);
  // A contiguous run of refills per warp (the counter cache's upper part lasts 2,730 refills); warps are
  // dealt to the CTAs in turn, so that few refills spread over the SMs, where a warp alone is
  // three times as fast as one of 16.
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t run = ((total + warps - 1) / warps + 31u) & ~31u;
  if (blockIdx.x * run >= total) return;
  if (!aes_fill_tables(status)) return;
  __syncthreads();
  const AesCtx c = aes_ctx();
  uint32_t rk[60];
  uint32_t st = 0;
  uint32_t lo = 1, hi = 0;  // refill range of stream st (empty: forces the first lookup)
  CtrCache cc;
  const uint32_t g0 = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * run, g1 = min(total, g0 + run);
  for (uint32_t g = g0 + (threadIdx.x & 31u); g < g1; g += 32u) {
    if (g < lo || g >= hi) {
      st = seg_of_refill(sg, g);
      lo = (uint32_t)seg_roff(sg, st);
      hi = (uint32_t)seg_roff(sg, st + 1);
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

// Call c of a stream starts at a fresh refill a_c and ends with the first refill e whose inclusive
// count of accepted candidates reaches E(a_c) + n; a_{c+1} = e + 1.  call_start of stream st:
// coff[st] + st .. coff[st+1] + st (calls + 1 entries; the last is the end of the last call).
//
// Short runs: k_walk, below, one CTA per stream.  Many calls of few refills: pointer doubling (k_next and
// those after it).  Long runs: by the overshoot.  A call ends up to 7
// samples beyond its n, and call c ends where the count reaches (c + 1) n + s, s being the overshoot of the
// calls before it: a number close to c times its mean.  So the refill that ends call c can be
// written down beforehand for every s in a window around that (k_ends: every refill writes itself
// to the at most 8 thresholds that it reaches), and what remains serial is one table read per call
// (k_chain).  The table is W words per call; s outside of the window is searched for directly.
// 785 calls of n = 4096 from one stream: 3 + 10 + 54 us where scanning the counts and walking over them
// in memory took 124; of 40 streams: 12 + 108 + 54 against 731, the chain being bound by the latency of
// one step (a shared-memory read and ten instructions, 69 ns) and k_ends by its instructions.
struct EndTable {
  uint32_t *ends;   // [call][W]: refill | overshoot << 28
  uint32_t *counts; // [stream][max_tiles]: accepted candidates per tile
  uint32_t W, max_tiles, mean;  // mean overshoot, 16 fractional bits
};
constexpr int kCountTile = 4096;

// window of call c: s in [first, first + W), first negative (mod 2^32) in the first calls
__device__ __forceinline__ uint32_t window_first(const EndTable &t, uint32_t c) {
  return (uint32_t)(((uint64_t)t.mean * c) >> 16) - t.W / 2;
}

// accept counts of tile blockIdx.x of stream blockIdx.y
__global__ void __launch_bounds__(256)
    k_tile_counts(const uint8_t *__restrict__ amask, SegDev sg, uint32_t *__restrict__ counts, uint32_t max_tiles) {
  __shared__ uint32_t wsum[8];
  const uint64_t r0 = seg_roff(sg, blockIdx.y);
  const uint32_t R = (uint32_t)(seg_roff(sg, blockIdx.y + 1) - r0), at = blockIdx.x * kCountTile + threadIdx.x * 16;
  if (blockIdx.x * kCountTile >= R) return;
  uint32_t n = 0;
  if (at < R) {  // R and r0 are multiples of 32
    const uint4 m = __ldg(reinterpret_cast<const uint4 *>(amask + r0 + at));
    n = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31u) == 0) wsum[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t v = 0;
    for (int i = 0; i < 8; ++i) v += wsum[i];
    counts[(size_t)blockIdx.y * max_tiles + blockIdx.x] = v;
  }
}

// What a stream has accepted before this thread's 16 refills of tile blockIdx.x, and their masks m and count
// (256 threads; past: the counts of the stream's tiles; refills at .. at + 15 of R)
__device__ __forceinline__ uint32_t accepted_before(const uint8_t *amask, uint64_t r0, uint32_t R, uint32_t at,
                                                    const uint32_t *counts, uint4 &m, uint32_t &own) {
  __shared__ uint32_t wsum[8], psum[8];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t past = 0;
  for (uint32_t i = threadIdx.x; i < blockIdx.x; i += 256) past += __ldg(counts + i);
  m = make_uint4(0, 0, 0, 0);
  if (at < R) m = __ldg(reinterpret_cast<const uint4 *>(amask + r0 + at));
  own = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
  uint32_t inc = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += v;
  }
  past = __reduce_add_sync(0xffffffffu, past);
  if (lane == 0) psum[warp] = past;
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint32_t E = inc - own;
#pragma unroll
  for (uint32_t i = 0; i < 8; ++i) E += psum[i] + (i < warp ? wsum[i] : 0u);
  return E;
}

// the table entries that the refills of tile blockIdx.x of stream blockIdx.y reach
__global__ void __launch_bounds__(256) k_ends(const uint8_t *__restrict__ amask, SegDev sg, EndTable t) {
  const uint32_t st = blockIdx.y;
  const uint64_t r0 = seg_roff(sg, st);
  const uint32_t R = (uint32_t)(seg_roff(sg, st + 1) - r0), at = blockIdx.x * kCountTile + threadIdx.x * 16;
  if (blockIdx.x * kCountTile >= R) return;
  uint4 m;
  uint32_t own;
  uint32_t E = accepted_before(amask, r0, R, at, t.counts + (size_t)st * t.max_tiles, m, own);
  // thresholds (c + 1) n + s in (E, E + own], c the call whose window they can lie in (end_table_width)
  const uint32_t n = seg_n(sg, st), calls = seg_calls(sg, st);
  // c + 1 to the nearest, (c + 1) (n + mean) - mean being the middle of call c's window
  const double mean = (double)t.mean / 65536.0, inv = 1.0 / ((double)n + mean);
  const uint32_t c1 = (uint32_t)(((double)(E + own / 2) + mean) * inv + 0.5);
  if (c1 == 0 || c1 > calls || own == 0) return;
  const uint32_t c = c1 - 1, lo = c1 * n + window_first(t, c), hi = lo + t.W;
  if (E + own < lo || E >= hi) return;
  uint32_t *row = t.ends + (seg_coff(sg, st) + c) * t.W;
  const uint32_t w[4] = {m.x, m.y, m.z, m.w};
#pragma unroll 1
  for (uint32_t i = 0; i < 16; ++i) {
    const uint32_t to = E + __popc((w[i >> 2] >> (8 * (i & 3u))) & 0xffu);
    if (to >= lo && E < hi) {
#pragma unroll
      for (uint32_t j = 1; j <= 8; ++j) {
        const uint32_t x = E + j;
        if (x <= to && x >= lo && x < hi) row[x - lo] = (at + i) | ((to - x) << 28);
      }
    }
    E = to;
  }
}

// One CTA per stream follows the table.  Warp 0 makes the steps, about ten instructions each, since a warp
// alone issues one in four or five cycles; the others copy the rows of 16 calls to shared memory three
// groups of calls ahead, 128 entries each around the s that is expected there.  A group in which s
// left a copied row is made again with reads of the table, and outside of the window by a search.
constexpr uint32_t kChainRows = 16, kChainAhead = 4, kChainCols = 128;
__global__ void __launch_bounds__(128)
    k_chain(const uint8_t *__restrict__ amask, SegDev sg, EndTable t, uint32_t *__restrict__ call_start,
            uint32_t *__restrict__ status) {
  __shared__ __align__(16) uint32_t ring[kChainAhead][kChainRows][kChainCols];
  __shared__ uint32_t low[kChainAhead][kChainRows];  // the s of a copied row's first entry
  __shared__ uint32_t now;                           // s at the start of the walker's group
  const uint32_t st = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t n = seg_n(sg, st), calls = seg_calls(sg, st), groups = (calls + kChainRows - 1) / kChainRows;
  const uint32_t *ends = t.ends + seg_coff(sg, st) * t.W;
  // the copies of group g, from the overshoot s before call c
  const auto copy = [&](uint32_t g, uint32_t s, uint32_t c) {
    for (uint32_t i = warp - 1; i < kChainRows; i += 3) {
      const uint32_t r = g * kChainRows + i;
      if (r >= calls) break;
      const uint32_t expect = s + (uint32_t)(((uint64_t)t.mean * (r - c)) >> 16), first = window_first(t, r);
      const int off = (int)(expect - first) - (int)(kChainCols / 2);
      const uint32_t from = min(off > 0 ? (uint32_t)off & ~3u : 0u, t.W - kChainCols);
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&ring[g % kChainAhead][i][4 * lane]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(ends + (size_t)r * t.W + from + 4 * lane)
                   : "memory");
      if (lane == 0) low[g % kChainAhead][i] = first + from;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (threadIdx.x == 0) now = 0;
  if (warp) {
    for (uint32_t g = 0; g + 1 < kChainAhead; ++g) copy(g, 0, 0);
    asm volatile("cp.async.wait_group %0;" ::"n"(kChainAhead - 2) : "memory");
    __syncthreads();
    for (uint32_t g = 0; g < groups; ++g) {
      copy(g + kChainAhead - 1, now, g * kChainRows);
      asm volatile("cp.async.wait_group %0;" ::"n"(kChainAhead - 2) : "memory");  // group g + 1 is there
      __syncthreads();
      if (__syncthreads_or(0)) break;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return;
  }
  const uint64_t r0 = seg_roff(sg, st);
  const uint32_t R = (uint32_t)(seg_roff(sg, st + 1) - r0), tiles = (R + kCountTile - 1) / kCountTile;
  const uint32_t *counts = t.counts + (size_t)st * t.max_tiles;
  uint32_t *cs = call_start + seg_coff(sg, st) + st;
  uint32_t total = 0;
  for (uint32_t i = lane; i < tiles; i += 32) total += __ldg(counts + i);
  total = __reduce_add_sync(0xffffffffu, total);
  uint32_t s = 0, a = 0, c = 0;  // overshoot so far, start refill of call c
  bool bad = false;
  __syncthreads();
  for (uint32_t g = 0; g < groups; ++g) {
    const uint32_t rows = min(kChainRows, calls - c), s0 = s, a0 = a;
    const uint32_t(*rg)[kChainCols] = ring[g % kChainAhead];
    const uint32_t *lw = low[g % kChainAhead];
    uint32_t worst = 0;
    // every threshold of a whole group within the stream's count: the short steps
    bool slow = rows < kChainRows || (uint64_t)(c + kChainRows) * n + s + 8 * kChainRows > total;
    if (!slow) {
#pragma unroll
      for (uint32_t i = 0; i < kChainRows; ++i) {
        const uint32_t in = s - lw[i];
        worst = max(worst, in);
        const uint32_t end = rg[i][min(in, kChainCols - 1)];
        if (lane == 0) cs[c + i] = a;
        a = (end & 0x0fffffffu) + 1u;
        s += end >> 28;
      }
      slow = worst >= kChainCols;
      if (!slow) c += kChainRows;
    }
    if (slow) {
      s = s0;
      a = a0;
      for (uint32_t i = 0; i < rows; ++i) {
        const uint32_t x = (c + 1) * n + s, col = s - window_first(t, c);
        if (x > total) {  // the refill range was too short
          bad = true;
          break;
        }
        uint32_t end;
        if (col < t.W) {
          end = __ldg(ends + (size_t)c * t.W + col);
        } else {  // the tile, then the refill that reaches the threshold
          uint32_t E = 0, k = 0;
          while (k + 1 < tiles && E + __ldg(counts + k) < x) E += __ldg(counts + k++);
          for (uint32_t e = k * kCountTile;; e += 32) {  // total >= x: some refill below R reaches it
            const uint32_t own = e + lane < R ? __popc((uint32_t)__ldg(amask + r0 + e + lane)) : 0u;
            uint32_t inc = own;
            for (int o = 1; o < 32; o <<= 1) {
              const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
              if (lane >= (uint32_t)o) inc += v;
            }
            const uint32_t hit = __ballot_sync(0xffffffffu, E + inc >= x);
            if (hit || e >= R) {
              const uint32_t f = hit ? (uint32_t)__ffs(hit) - 1u : 31u;
              end = (e + f) | ((E + __shfl_sync(0xffffffffu, inc, f) - x) << 28);
              break;
            }
            E += __shfl_sync(0xffffffffu, inc, 31);
          }
        }
        if (lane == 0) cs[c] = a;
        a = (end & 0x0fffffffu) + 1u;
        s += end >> 28;
        ++c;
      }
    }
    __syncthreads();  // the copiers have read `now`
    if (lane == 0) now = s;
    if (__syncthreads_or(bad)) break;
  }
  if (lane == 0) {
    if (bad) atomicOr(status, kStatusRefillsExhausted);
    for (uint32_t i = c; i <= calls; ++i) cs[i] = bad ? R : a;
  }
}

// One CTA per stream, for runs of few calls or small n.
//
// The stream is serial in its calls, so one warp walks; the other eight stream the accept masks
// ahead of it, 8,192 refills at a time, and leave in shared memory the count before every 16
// refills and the counts within them.  A call then costs the walker one round of reads around its
// expected end, a ballot and a shuffle, whatever n is, and no count goes through memory.  (Walked over
// prefixes in global memory a call cost 0.85 us of dependent loads.)
constexpr int kWalkTile = 8192, kWalkGroups = kWalkTile / 16;
constexpr int kWalkThreads = 32 + 256;  // the walker, and 32 refills per thread
__global__ void __launch_bounds__(kWalkThreads)
    k_walk(const uint8_t *__restrict__ amask, SegDev sg, float mean_accept, uint32_t *__restrict__ call_start,
           uint32_t *__restrict__ status) {
  __shared__ uint32_t before[2][kWalkGroups + 1];         // E at the groups' starts and the tile's end
  __shared__ __align__(16) uint8_t within[2][kWalkTile];  // inclusive count within the group (at most 128)
  __shared__ uint32_t wsum[2][8];
  const uint32_t st = blockIdx.x, lane = threadIdx.x & 31u;
  const uint64_t r0 = seg_roff(sg, st);
  const uint32_t R = (uint32_t)(seg_roff(sg, st + 1) - r0);  // a multiple of 32, as every r0
  const uint32_t tiles = (R + kWalkTile - 1) / kWalkTile;
  if (threadIdx.x >= 32) {
    const uint32_t g = threadIdx.x - 32, warp = g >> 5;
    const uint4 *src = reinterpret_cast<const uint4 *>(amask + r0) + 2 * g;
    const auto load = [&](uint32_t tile, uint4 (&m)[2]) {
      const bool in = tile * kWalkTile + 32 * g < R;
      m[0] = in ? __ldg(src + (size_t)tile * kWalkGroups) : make_uint4(0, 0, 0, 0);
      m[1] = in ? __ldg(src + (size_t)tile * kWalkGroups + 1) : make_uint4(0, 0, 0, 0);
    };
    // 16 masks to the inclusive counts up to each; returns the sum
    const auto count = [](uint4 m, uint8_t *to) {
      uint32_t w[4] = {m.x, m.y, m.z, m.w}, run = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // bytes to their bit counts, then to the sums up to each byte
        uint32_t v = w[i] - ((w[i] >> 1) & 0x55555555u);
        v = (v & 0x33333333u) + ((v >> 2) & 0x33333333u);
        v = (v + (v >> 4)) & 0x0f0f0f0fu;
        w[i] = (v + run) * 0x01010101u;  // at most 128 each
        run = w[i] >> 24;
      }
      *reinterpret_cast<uint4 *>(to) = make_uint4(w[0], w[1], w[2], w[3]);
      return run;
    };
    uint32_t carry = 0;
    uint4 m[2], m1[2];  // two tiles of loads in flight
    load(0, m);
    load(1, m1);
    for (uint32_t k = 0; k <= tiles; ++k) {
      if (k < tiles) {
        const uint32_t buf = k & 1u;
        const uint32_t c0 = count(m[0], &within[buf][32 * g]), c1 = count(m[1], &within[buf][32 * g + 16]);
        m[0] = m1[0], m[1] = m1[1];
        load(k + 2, m1);
        uint32_t inc = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= (uint32_t)o) inc += v;
        }
        if (lane == 31) wsum[buf][warp] = inc;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        uint32_t base = carry;
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
          const uint32_t v = wsum[buf][i];
          if (i < warp) base += v;
          carry += v;
        }
        before[buf][2 * g] = base + inc - c0 - c1;
        before[buf][2 * g + 1] = base + inc - c1;
        if (g == 255) before[buf][kWalkGroups] = carry;
      }
      if (__syncthreads_or(0)) return;  // the walker has every call
    }
    return;
  }
  const uint32_t n = seg_n(sg, st), calls = seg_calls(sg, st);
  const uint32_t guess = (uint32_t)((float)n / mean_accept);
  uint32_t *cs = call_start + seg_coff(sg, st) + st;
  uint32_t a = 0, c = 0, target = n;  // start refill of call c, E(a) + n
  if (lane == 0 && calls) cs[0] = 0;
  __syncthreads_or(0);  // tile 0 is there
  for (uint32_t k = 0; k < tiles; ++k) {
    const uint32_t *bf = before[k & 1u];
    const uint32_t *in = reinterpret_cast<const uint32_t *>(within[k & 1u]) + lane;
    const uint32_t t0 = k * kWalkTile, tile_end = bf[kWalkGroups];
    // 128 refills around refill a + span, four per lane
    const auto window = [&](uint32_t span) {
      const uint32_t at = a + span > t0 + 64 ? a + span - t0 - 64 : 0u;
      return min(at & ~3u, (uint32_t)kWalkTile - 128);
    };
    const auto base = [&](uint32_t w) { return bf[((w >> 2) + lane) >> 2]; };
    uint32_t w = window(guess), v = in[w >> 2], e = base(w);
    while (c < calls && tile_end >= target) {
      // the next call's window is read while this call is decided
      const uint32_t w1 = window(2 * guess), v1 = in[w1 >> 2], e1 = base(w1);
      uint32_t first, mine;
      for (;;) {
        const int32_t left = (int32_t)(target - e);
        // refills of these four that do not reach the target, and how far the next one goes beyond it
        const uint32_t cnt = (uint32_t)((int32_t)(v & 0xffu) < left) + (uint32_t)((int32_t)((v >> 8) & 0xffu) < left) +
                             (uint32_t)((int32_t)((v >> 16) & 0xffu) < left) + (uint32_t)((int32_t)(v >> 24) < left);
        const uint32_t hit = __ballot_sync(0xffffffffu, cnt < 4);
        mine = cnt | ((uint32_t)((int32_t)((v >> (8 * (cnt & 3u))) & 0xffu) - left) << 2);
        first = (uint32_t)__ffs(hit) - 1u;
        mine = __shfl_sync(0xffffffffu, mine, first & 31u);
        if (hit && (first | (mine & 3u) | (uint32_t)(w == 0))) break;
        // outside of the window; reached in its first refill, the call may have ended before it
        w = hit ? (w > 124 ? w - 124 : 0u) : min(w + 128, (uint32_t)kWalkTile - 128);
        v = in[w >> 2];
        e = base(w);
      }
      a = t0 + w + 4 * first + (mine & 3u) + 1u;
      target += (mine >> 2) + n;
      ++c;
      if (lane == 0) cs[c] = a;
      w = w1, v = v1, e = e1;
    }
    if (__syncthreads_or(c >= calls)) return;
  }
  if (c < calls && lane == 0) {  // the refill range was too short
    atomicOr(status, kStatusRefillsExhausted);
    for (uint32_t i = c; i <= calls; ++i) cs[i] = R;
  }
}

// Pointer doubling, for runs whose calls are many and their refills few: the walk and the table take a
// step per call of the longest stream, this one log2(calls) launches over all refills.  next(t) is the refill
// after a call that starts at refill t, R + 1 where the stream runs out; call c starts where next applied c
// times to 0 leads, from the bits of c with the tables next^(2^k).
//
// counts of accepted candidates up to and with each refill of tile blockIdx.x of stream blockIdx.y
__global__ void __launch_bounds__(256)
    k_prefix(const uint8_t *__restrict__ amask, SegDev sg, const uint32_t *__restrict__ counts, uint32_t max_tiles,
             uint32_t *__restrict__ upto) {
  const uint64_t r0 = seg_roff(sg, blockIdx.y);
  const uint32_t R = (uint32_t)(seg_roff(sg, blockIdx.y + 1) - r0), at = blockIdx.x * kCountTile + threadIdx.x * 16;
  if (blockIdx.x * kCountTile >= R) return;
  uint4 m;
  uint32_t own;
  uint32_t E = accepted_before(amask, r0, R, at, counts + (size_t)blockIdx.y * max_tiles, m, own);
  if (at >= R) return;
  const uint32_t w[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 v;
    v.x = E += __popc(w[i] & 0xffu);
    v.y = E += __popc(w[i] & 0xff00u);
    v.z = E += __popc(w[i] & 0xff0000u);
    v.w = E += __popc(w[i] & 0xff000000u);
    reinterpret_cast<uint4 *>(upto + r0 + at)[i] = v;
  }
}

__global__ void __launch_bounds__(256) k_next(const uint32_t *__restrict__ upto, SegDev sg, float mean_accept,
                                              uint32_t *__restrict__ next) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (uint32_t)seg_roff(sg, sg.nstreams)) return;
  const uint32_t st = seg_of_refill(sg, g), n = seg_n(sg, st);
  const uint64_t r0 = seg_roff(sg, st);
  const uint32_t R = (uint32_t)(seg_roff(sg, st + 1) - r0), t = g - (uint32_t)r0;
  const uint32_t *up = upto + r0;
  const uint32_t target = (t ? up[t - 1] : 0u) + n;
  // the first e >= t with up[e] >= target; twice the expected length first
  uint32_t lo = t, hi = R;
  const uint32_t guess = t + 2u * (uint32_t)((float)n / mean_accept) + 64u;
  if (guess < R && up[guess] >= target) hi = guess;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (up[mid] >= target) hi = mid;
    else lo = mid + 1;
  }
  next[g] = lo < R ? lo + 1 : R + 1;
}

__global__ void __launch_bounds__(256)
    k_next_square(const uint32_t *__restrict__ in, uint32_t *__restrict__ out, SegDev sg) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (uint32_t)seg_roff(sg, sg.nstreams)) return;
  const uint32_t st = seg_of_refill(sg, g);
  const uint64_t r0 = seg_roff(sg, st);
  const uint32_t R = (uint32_t)(seg_roff(sg, st + 1) - r0), a = in[g];
  out[g] = a < R ? in[r0 + a] : R + 1;
}

// one thread per entry of call_start, c = 0 .. calls of every stream
__global__ void __launch_bounds__(256)
    k_doubled_starts(const uint32_t *__restrict__ tables, uint32_t levels, uint64_t stride, SegDev sg,
                     uint32_t *__restrict__ call_start, uint32_t *__restrict__ status) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= seg_coff(sg, sg.nstreams) + sg.nstreams) return;
  uint32_t lo = 0, hi = sg.nstreams;  // stream s has the entries from coff[s] + s on
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (seg_coff(sg, mid) + mid <= i) lo = mid;
    else hi = mid;
  }
  const uint32_t c = (uint32_t)(i - (seg_coff(sg, lo) + lo));
  const uint64_t r0 = seg_roff(sg, lo);
  const uint32_t R = (uint32_t)(seg_roff(sg, lo + 1) - r0);
  uint32_t a = 0;
  for (uint32_t k = 0; k < levels; ++k)
    if ((c >> k) & 1u) a = a < R ? tables[k * stride + r0 + a] : R + 1;
  call_start[i] = min(a, R);
  if (a > R && c == seg_calls(sg, lo)) atomicOr(status, kStatusRefillsExhausted);
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
// consecutive output positions.  The first position of a warp's run is the accept count of the
// runs before it, which the warps count first.
constexpr int kScatterThreads = 256;
__global__ void __launch_bounds__(kScatterThreads)
    k_scatter(const uint32_t *__restrict__ cand_lo, const uint8_t *__restrict__ amask,
              const uint16_t *__restrict__ chs, const uint32_t *__restrict__ call_start, SegDev sg, ModArgs m,
              uint32_t *__restrict__ out) {
  __shared__ uint2 stage[kScatterThreads / 32][256];
  __shared__ uint32_t counts[kScatterThreads / 32];
  const uint32_t st = seg_of_call(sg, blockIdx.x);
  const uint64_t cs0 = seg_coff(sg, st), r0 = seg_roff(sg, st);
  const uint32_t c = (uint32_t)(blockIdx.x - cs0), R = (uint32_t)(seg_roff(sg, st + 1) - r0);
  const uint32_t n = seg_n(sg, st);
  const uint32_t *cs = call_start + cs0 + st;
  const uint32_t a = cs[c], b = min(cs[c + 1], R);
  if (a >= b) return;
  constexpr uint32_t nw = kScatterThreads / 32;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t span = ((b - a + nw - 1) / nw + 3u) & ~3u;  // refills per warp
  const uint32_t t0 = min(a + warp * span, b), t1 = min(t0 + span, b);
  uint32_t mine = 0;
#pragma unroll 4
  for (uint32_t t = t0 + lane; t < t1; t += 32) mine += __popc((uint32_t)__ldg(amask + r0 + t));
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) counts[warp] = mine;
  __syncthreads();
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t i = 0; i < nw; ++i) pos += i < warp ? counts[i] : 0u;
  uint32_t *o = out + seg_ooff(sg, st) + (size_t)c * 3 * n;
  uint2 *sw = stage[warp];
  const uint32_t below = (1u << lane) - 1u, ci = lane & 7u;
  for (uint32_t t = t0; t < t1 && pos < n; t += 32) {
    // refill t + lane: accept bits, bit 32 of each |value| (<< 8), signs (<< 16)
    const uint32_t mk = t + lane < t1 ? (uint32_t)__ldg(amask + r0 + t + lane) |
                                            ((uint32_t)__ldg(chs + r0 + t + lane) << 8)
                                      : 0u;
    uint32_t lv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t r = t + 4 * k + (lane >> 3);
      lv[k] = r < t1 ? __ldg(cand_lo + (r0 + r) * 8 + ci) : 0u;
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
  if (!aes_fill_tables(status)) return;
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
                                               uint32_t *__restrict__ a, uint32_t *__restrict__ status) {
  if (!aes_fill_tables(status)) return;
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
// Mean samples by which a call overshoots its n, with 16 fractional bits: (E[X^2] / E[X] - 1) / 2 for
// the accept count X of a refill with the moments above: 2.38, 1.92 and 1.35.
static uint32_t mean_overshoot(int sig) { return sig == 0 ? 156100u : (sig == 1 ? 126000u : 88500u); }

// Refills precomputed for `calls` consecutive calls of n samples.  A call consumes r refills,
// the first whose accepted total reaches n; E[r] = (n + overshoot) / mu < n / mu + 1 (the
// overshoot averages less than half of mu: mean_overshoot), and over many calls sum(r) has variance about
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
  SegDev d{};
  d.nstreams = S;
  d.n = reinterpret_cast<const uint32_t *>(b + L.n);
  d.calls = reinterpret_cast<const uint32_t *>(b + L.calls);
  d.roff = reinterpret_cast<const uint64_t *>(b + L.roff);
  d.coff = reinterpret_cast<const uint64_t *>(b + L.coff);
  d.ooff = reinterpret_cast<const uint64_t *>(b + L.ooff);
  return d;
}

// Width of the table of call ends, 0: not possible.  The overshoot of a call has a standard deviation
// below 2, so that of c calls one below 2 sqrt(c): the window takes 4 of those and 64 to either side.  The
// windows may be n - 192 wide, so that a threshold is in one of them, and the nearest call to
// any of a thread's 128 thresholds is the one whose window it is in (k_ends).
static uint32_t end_table_width(const SegSizes &z) {
  const uint32_t W = ((uint32_t)(16.0 * std::sqrt((double)z.max_calls)) + 128 + 63) & ~63u;
  return W + 192 <= z.min_n && z.max_refills < (1u << 28) && z.nstreams < 65536u ? W : 0u;
}

static uint32_t doubling_levels(const SegSizes &z) {
  uint32_t k = 1;
  while (k < 31 && (1u << k) <= z.max_calls) ++k;
  return k;  // bit length of max_calls
}
static bool doubling_ok(const SegSizes &z) { return z.refills <= ((uint64_t)32 << 20) && z.nstreams < 65536u; }

bool seg_search(SegSizes &z, CallSearch how) {
  const uint32_t w = how == kSearchTable ? end_table_width(z) : 0u;
  if ((how == kSearchTable && !w) || (how == kSearchDoubling && !doubling_ok(z))) return false;
  z.search = how;
  z.end_w = w;
  z.end_mean = 1;
  return true;
}

static std::atomic<int> g_call_search{0};
void set_call_search(int mode) { g_call_search = mode; }

// The search of a run: the one that cufe_sampler_call_search asked for, or by time.  From 128 calls on the
// table's three launches are shorter than the walk.  Doubling takes over where it is at most 3/4 of the other by
// these estimates, us on a B200, within 25% of what they were fitted to (n 16..8192, 1..40 streams, 16..16,000
// calls); by less it is not worth its tables, 4 bytes per refill and level.  Measured, walk | table |
// doubling, sigma_3 of one stream: n = 4096, 64 calls 19 | 22 | 46, 128 31 | 27 | 50, 784 158 | 72 | 87; n = 512,
// 256 calls 46 | - | 52, 512 84 | - | 58, 784 125 | - | 57, 4,000 617 | - | 89; n = 1024, 1,024 calls 168 | 89 | 64,
// 4,000 639 | - | 117; n = 2048, 4,000 calls 684 | 312 | 162; n = 512, 8 streams of 784 calls 126 | - | 84, 40 of
// them 128 | - | 232.
static void choose_search(SegSizes &z) {
  const int mode = g_call_search;
  seg_search(z, kSearchWalk);
  if (mode == 1) return;
  const double calls = z.max_calls, refills = (double)z.refills;
  double best = 6.0 + 0.146 * calls + 37e-6 * z.max_refills;
  if (mode == 0 && z.max_calls >= 128 && seg_search(z, kSearchTable)) best = 17.0 + 0.078 * calls + 1.4e-6 * refills;
  if (mode == 2 || 18.0 + doubling_levels(z) * (3.4 + 3.6e-6 * refills) < 0.75 * best) seg_search(z, kSearchDoubling);
}

SegSizes seg_fill_host(int sig, uint32_t S, const uint32_t *calls, const uint32_t *n, const uint64_t *ooff,
                       void *host_base) {
  const SegLayout L = seg_layout(S);
  uint8_t *b = static_cast<uint8_t *>(host_base);
  uint32_t *hn = reinterpret_cast<uint32_t *>(b + L.n), *hc = reinterpret_cast<uint32_t *>(b + L.calls);
  uint64_t *hr = reinterpret_cast<uint64_t *>(b + L.roff), *hco = reinterpret_cast<uint64_t *>(b + L.coff);
  uint64_t *ho = reinterpret_cast<uint64_t *>(b + L.ooff);
  SegSizes z{S, 0, 0, 0, 0, 0xffffffffu, kSearchWalk, 0, 1};
  for (uint32_t i = 0; i < S; ++i) {
    const uint32_t R = cpu_map_refills(calls[i], n[i], sig);
    hn[i] = n[i];
    hc[i] = calls[i];
    ho[i] = ooff ? ooff[i] : 0;
    hr[i] = z.refills;
    hco[i] = z.calls;
    z.refills += R;
    z.max_refills = std::max(z.max_refills, R);
    z.max_calls = std::max(z.max_calls, calls[i]);
    z.min_n = std::min(z.min_n, n[i]);
    z.calls += calls[i];
  }
  hr[S] = z.refills;
  hco[S] = z.calls;
  choose_search(z);
  return z;
}

SegSizes cpu_map_sizes(uint32_t S, uint32_t calls, uint32_t n, int sig) {
  const uint32_t R = cpu_map_refills(calls, n, sig);
  SegSizes z{S, (uint64_t)S * R, (uint64_t)S * calls, R, calls, n, kSearchWalk, 0, 1};
  choose_search(z);
  return z;
}

static uint32_t count_tiles(const SegSizes &z) { return (z.max_refills + kCountTile - 1) / kCountTile; }

size_t seg_scratch_bytes(const SegSizes &z) {
  size_t b = align256(z.refills * 32) + align256(z.refills) + align256(z.refills * 2) +
             align256((z.calls + z.nstreams) * 4);
  if (z.search != kSearchWalk) b += align256((size_t)z.nstreams * count_tiles(z) * 4);
  if (z.search == kSearchTable) b += align256((size_t)z.calls * z.end_w * 4);
  if (z.search == kSearchDoubling) b += (1 + (size_t)doubling_levels(z)) * align256(z.refills * 4);
  return b;
}

int sample_cpu_map_seg(int sig, const SegDev &sg, const SegSizes &z, const uint32_t *d_rkeys, uint32_t *d_out,
                       void *scratch, uint32_t *d_status, int num_sms, cudaStream_t s, int parts) {
  if (sig < 0 || sig > 2 || z.nstreams == 0 || z.calls >= (1ull << 31) ||
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
  uint32_t *cstart = reinterpret_cast<uint32_t *>(take((z.calls + z.nstreams) * 4));
  const double kinv = kinv_of(sig);
  const uint32_t grid =
      (uint32_t)std::min<uint64_t>((uint64_t)num_sms, (z.refills + 31) / 32);
  if (grid > 0 && (parts & kSampleCandidates)) {
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
  if (!(parts & kSampleRest)) return CUFE_OK;
  {
    ProfScope ps("sample_walk", s);
    const dim3 tiles(count_tiles(z), z.nstreams);
    if (z.search == kSearchTable) {
      EndTable t;
      t.ends = reinterpret_cast<uint32_t *>(take((size_t)z.calls * z.end_w * 4));
      t.max_tiles = tiles.x;
      t.counts = reinterpret_cast<uint32_t *>(take((size_t)z.nstreams * tiles.x * 4));
      t.W = z.end_w;
      t.mean = z.end_mean * mean_overshoot(sig);
      note_launch(), k_tile_counts<<<tiles, 256, 0, s>>>(amask, sg, t.counts, tiles.x);
      note_launch(), k_ends<<<tiles, 256, 0, s>>>(amask, sg, t);
      note_launch(), k_chain<<<z.nstreams, 128, 0, s>>>(amask, sg, t, cstart, d_status);
    } else if (z.search == kSearchDoubling) {
      uint32_t *counts = reinterpret_cast<uint32_t *>(take((size_t)z.nstreams * tiles.x * 4));
      uint32_t *upto = reinterpret_cast<uint32_t *>(take(z.refills * 4));
      const uint32_t levels = doubling_levels(z), grid = (uint32_t)((z.refills + 255) / 256);
      const uint64_t stride = align256(z.refills * 4) / 4;
      uint32_t *tab = reinterpret_cast<uint32_t *>(take(levels * stride * 4));
      note_launch(), k_tile_counts<<<tiles, 256, 0, s>>>(amask, sg, counts, tiles.x);
      note_launch(), k_prefix<<<tiles, 256, 0, s>>>(amask, sg, counts, tiles.x, upto);
      note_launch(), k_next<<<grid, 256, 0, s>>>(upto, sg, (float)mean_accept(sig), tab);
      for (uint32_t k = 1; k < levels; ++k)
        note_launch(), k_next_square<<<grid, 256, 0, s>>>(tab + (k - 1) * stride, tab + k * stride, sg);
      note_launch(), k_doubled_starts<<<(uint32_t)((z.calls + z.nstreams + 255) / 256), 256, 0, s>>>(tab, levels, stride, sg,
                                                                                                 cstart, d_status);
    } else {
      note_launch(), k_walk<<<z.nstreams, kWalkThreads, 0, s>>>(amask, sg, (float)mean_accept(sig), cstart, d_status);
    }
    CUFE_CUDA(cudaGetLastError());
  }
  if (d_out && z.calls) {
    ProfScope ps_sc("sample_scatter", s);
    note_launch(), k_scatter<<<(uint32_t)z.calls, kScatterThreads, 0, s>>>(cand, amask, chs, cstart, sg, mod_args(),
                                                                           d_out);
    CUFE_CUDA(cudaGetLastError());
  }
  return CUFE_OK;
}

// the uniform case: equal streams, no tables
int sample_cpu_map(int sig, const SegSizes &z, const uint32_t *d_rkeys, uint32_t *d_out, void *ws, uint32_t *d_status,
                   int num_sms, cudaStream_t s, uint32_t *d_out1, int parts) {
  if (z.max_refills >= (1ull << 32) / 24) return CUFE_ERR_INVALID;  // AES counter range
  if (d_out1 && z.nstreams != 2) return CUFE_ERR_INVALID;
  SegDev sg{};
  sg.nstreams = z.nstreams;
  sg.u_n = z.min_n;
  sg.u_calls = z.max_calls;
  sg.u_refills = z.max_refills;
  sg.u_ostride = (uint64_t)z.max_calls * 3 * z.min_n;
  if (d_out1)  // two streams: the distance between their outputs, wherever they lie
    sg.u_ostride = (uint64_t)((reinterpret_cast<intptr_t>(d_out1) - reinterpret_cast<intptr_t>(d_out)) / 4);
  return sample_cpu_map_seg(sig, sg, z, d_rkeys, d_out, ws, d_status, num_sms, s, parts);
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

int sample_polya(const uint32_t *d_rkey, uint32_t n, uint32_t *d_a, uint32_t *d_status, cudaStream_t s) {
  const uint32_t grid = (n / 2 + 255) / 256;
  ProfScope ps("sample_polya", s);
  note_launch(), k_polya<<<grid, 256, kAesSmemBytes, s>>>(d_rkey, n, mod_args(), d_a, d_status);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

}  // namespace cufe

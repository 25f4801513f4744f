// mac.cu -- the l-sums of key generation and decryption:
//   out[z][k][m][j] = sum_{i < l} y[k][i] v[z][i][m][j] mod q_m
// for keys k, RNS moduli m and coefficients j, with v = msk (src/rlwe_sife.c:215-245) or the
// ciphertexts z (the sum of src/rlwe_sife.c:248-278).
//
// Two kernels.  k_mac_few streams v once per KCH keys and is bound by memory; k_mac_mma is the
// product of many keys with v on the tensor cores.  Before, every product was three integer
// instructions and v was read once per 4 keys (key generation) or per key (decryption).  B200,
// us per call, before -> now: 1 key at n = 4096, l = 784 277 -> 16; 591 keys at l = 785 2034 -> 70;
// the decryption of one ciphertext under 591 keys at n = 2048, l = 124 254 -> 100.
#include <algorithm>

#include "ctx.h"
#include "prof.h"
#include "scheme.cuh"
#include "umma.cuh"

namespace cufe {

namespace {

// ------------------------------------------------------------------ few keys

constexpr int kFewThreads = 256;
constexpr int kFewRows = 1024;  // rows of y staged at a time

// An exact sum of products of a word and a residue below 2^31: two products at a time (below
// 2^64), folded into 64 + 32 bits.
struct WideSum {
  uint64_t lo = 0;
  uint32_t hi = 0;
  __device__ __forceinline__ void add(uint64_t t) {
    lo += t;
    hi += lo < t;
  }
  __device__ __forceinline__ uint32_t mod(uint64_t mu, uint32_t q) const {
    const uint64_t c64 = 0ull - mu * q;  // 2^64 mod q
    return mod_u64(mod_u64(lo, mu, q) + (uint64_t)hi * c64, mu, q);
  }
};

// Four consecutive words; vec: p is 16-byte aligned.
__device__ __forceinline__ uint4 load4(const uint32_t *p, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const uint4 *>(p));
  return make_uint4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
__device__ __forceinline__ void store4(uint32_t *p, uint4 v, bool vec) {
  if (vec) {
    *reinterpret_cast<uint4 *>(p) = v;
  } else {
    p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
  }
}

// A CTA sums 4 * lanes coefficients of one (z, modulus) for KCH keys: thread (slice, lane) takes 4
// coefficients (16-byte loads) of the rows slice, slice + slices, ..., eight rows in flight, and
// the slices are added in shared memory, so no partial sums go through memory.  Keys whose
// entries are all below 2^15 in magnitude (every quantised weight is) take one 64-bit
// multiply-add per product: with y + 2^15 in place of a signed y the sums stay below
// 2^32 2^16 l <= 2^64, and 2^15 times the sum of the words comes off at the end.  Others take
// their residues and the 96-bit sum.
template <int KCH>
__global__ void __launch_bounds__(kFewThreads)
    k_mac_few(const uint32_t *__restrict__ v, size_t vstride, const uint32_t *__restrict__ y, int y_signed, int nkeys,
              uint32_t *__restrict__ out, int lanes, int vec, SchemeArgs sa) {
  __shared__ uint32_t ys[KCH][kFewRows];
  __shared__ uint64_t red[kFewThreads][4];
  __shared__ uint32_t redh[kFewThreads][4];
  const int n = sa.ra.n, l = sa.l, tid = threadIdx.x;
  const int lane = tid & (lanes - 1), slice = tid / lanes, slices = kFewThreads / lanes;
  const int tiles = n / (4 * lanes);  // per residue polynomial
  const int m = blockIdx.x / tiles, j = 4 * ((blockIdx.x - m * tiles) * lanes + lane);
  const int z = blockIdx.y, k0 = blockIdx.z * KCH;
  const uint32_t q = sa.ra.q[m], bias = y_signed ? 32768u : 0u;
  const uint64_t mu = sa.mu[m];
  const uint32_t *vb = v + z * vstride + (size_t)m * n + j;
  const size_t row = (size_t)3 * n;
  bool big = false;
  for (int t = tid; t < KCH * l; t += kFewThreads) {
    const int kk = t / l;
    if (k0 + kk < nkeys) big |= y[(size_t)(k0 + kk) * l + (t - kk * l)] + bias > 65535u;
  }
  big = __syncthreads_or(big);
  uint64_t acc[KCH][4], sx[4];
  uint32_t hi[KCH][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    sx[e] = 0;
#pragma unroll
    for (int kk = 0; kk < KCH; ++kk) acc[kk][e] = 0, hi[kk][e] = 0;
  }
  for (int r0 = 0; r0 < l; r0 += kFewRows) {
    const int rows = min(kFewRows, l - r0);
    if (r0) __syncthreads();
    for (int t = tid; t < KCH * kFewRows; t += kFewThreads) {
      const int kk = t / kFewRows, i = t % kFewRows;
      uint32_t w = 0;
      if (i < rows && k0 + kk < nkeys) {
        w = y[(size_t)(k0 + kk) * l + r0 + i];
        w = big ? y_residue(w, y_signed, q, mu) : w + bias;
      }
      ys[kk][i] = w;
    }
    __syncthreads();
    const uint32_t *vr = vb + (size_t)r0 * row;
    for (int i = slice; i < rows; i += 8 * slices) {
      uint4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = i + u * slices;
        x[u] = r < rows ? load4(vr + (size_t)r * row, vec) : make_uint4(0, 0, 0, 0);
      }
      if (!big) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          sx[0] += x[u].x, sx[1] += x[u].y, sx[2] += x[u].z, sx[3] += x[u].w;
#pragma unroll
          for (int kk = 0; kk < KCH; ++kk) {
            const uint32_t yv = ys[kk][min(i + u * slices, kFewRows - 1)];
            acc[kk][0] += (uint64_t)x[u].x * yv;
            acc[kk][1] += (uint64_t)x[u].y * yv;
            acc[kk][2] += (uint64_t)x[u].z * yv;
            acc[kk][3] += (uint64_t)x[u].w * yv;
          }
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < KCH; ++kk)
#pragma unroll
          for (int u = 0; u < 8; u += 2) {
            const uint32_t y0 = ys[kk][min(i + u * slices, kFewRows - 1)];
            const uint32_t y1 = ys[kk][min(i + (u + 1) * slices, kFewRows - 1)];
            const uint64_t t[4] = {(uint64_t)x[u].x * y0 + (uint64_t)x[u + 1].x * y1,
                                   (uint64_t)x[u].y * y0 + (uint64_t)x[u + 1].y * y1,
                                   (uint64_t)x[u].z * y0 + (uint64_t)x[u + 1].z * y1,
                                   (uint64_t)x[u].w * y0 + (uint64_t)x[u + 1].w * y1};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              acc[kk][e] += t[e];
              hi[kk][e] += acc[kk][e] < t[e];
            }
          }
      }
    }
  }
  // add the slices of one key at a time (the bias first); the first `lanes` threads finish
#pragma unroll
  for (int kk = 0; kk < KCH; ++kk) {
    if (kk) __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      red[tid][e] = big ? acc[kk][e] : (uint64_t)mod_u64(acc[kk][e], mu, q) + (q - mod_u64(sx[e] * bias, mu, q));
      if (big) redh[tid][e] = hi[kk][e];
    }
    __syncthreads();
    if (tid < lanes && k0 + kk < nkeys) {
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        WideSum w;
        for (int s = 0; s < slices; ++s) {
          w.add(red[s * lanes + tid][e]);
          if (big) w.hi += redh[s * lanes + tid][e];
        }
        o[e] = w.mod(mu, q);
      }
      store4(out + ((size_t)(z * (size_t)nkeys + k0 + kk) * 3 + m) * n + j, make_uint4(o[0], o[1], o[2], o[3]), vec);
    }
  }
}

// ------------------------------------------------------------------ many keys

// The sums of 128 keys x 64 coefficients as an exact 8-bit integer product on the tensor cores.
// A: 128 keys x K signed bytes, the y of the CTA's key tile, packed once and resident in shared
// memory.  B: 256 rows x K unsigned bytes, the four bytes of 64 coefficients (row 64 b + c: byte b
// of coefficient c), built from v by byte transposes while it streams through two stages of 128
// slots.  The accumulators hold sum_i y_i byte_b(v_i), at most 128 * 255 * l < 2^31, and the
// epilogue puts the four together, reduces and stores.  CTAs are persistent: one key tile each,
// coefficient tiles in turn, the loads of the next two stages in flight.
//
// Inside a stage the byte position 4 t + i stands for slot 32 i + t (t < 32, i < 4): a warp then
// packs y from coalesced loads, and since A and B agree the order of the sum does not matter.
constexpr int kMmaThreads = 512;
constexpr int kMmaKeys = 128, kMmaCols = 64, kMmaK = 128;
constexpr uint32_t kMmaLboA = kMmaKeys * 16 + 16;  // the 16 spread the packing stores over the banks
constexpr uint32_t kMmaLboB = 4 * kMmaCols * 16;
constexpr uint32_t kMmaStage = kMmaK / 16 * kMmaLboB;
constexpr uint32_t kMmaTmem = 256;
constexpr int kMmaPitch = kMmaCols + 4;  // words per key of the staged output: conflict-free 16-byte accesses
static_assert(kMmaKeys * kMmaPitch * 4 <= 2 * kMmaStage, "the output fits the two stages");
constexpr int kMmaMaxL = 1280;  // A and two stages of B fit in 227 KB
constexpr uint32_t mma_smem(int l) {
  return (uint32_t)((l + kMmaK - 1) / kMmaK * (kMmaK / 16)) * kMmaLboA + 2 * kMmaStage + 64;
}
static_assert(mma_smem(kMmaMaxL) <= 232448, "shared memory of one CTA");
constexpr uint32_t kMmaIdesc = umma_i8_desc(true, 4 * kMmaCols);

struct MmaArgs {
  const uint32_t *v;
  size_t vstride;
  const uint32_t *y;
  int y_signed, nkeys, nz, key_tiles, vec;
  uint32_t *out;
  // Reduction of a sum s, |s| < 2^50 (l <= 1280): with off a multiple of q of at least 2^50 and below
  // 2^50 + 2^31, x = s + off is in [0, 2^51 + 2^31); its top (x >> 20, 32 bits) times
  // mul = floor(2^(52 + sh) / q) (32 bits) gives floor(x / q) or one less, since the cut-off bits
  // are below 2^20 < q / 8 and the rounding of mul below 2^-10.
  uint64_t off[3];
  uint32_t mul[3];
  int sh[3];
};

// The same tiles for keys with entries outside a signed byte: 96-bit sums of residue products,
// 16 keys per thread, y staged 32 slots at a time.
__device__ __noinline__ void mac_tiles_general(const MmaArgs &a, const SchemeArgs &sa, uint32_t *ystage, int key0,
                                               int first, int stride, int tiles) {
  constexpr int KS = 32, PITCH = kMmaKeys + 4;
  const int n = sa.ra.n, l = sa.l, per_z = 3 * n / kMmaCols;
  const int c = threadIdx.x & (kMmaCols - 1), kg = threadIdx.x / kMmaCols;
  for (int tile = first; tile < tiles; tile += stride) {
    const int z = tile / per_z, col = (tile - z * per_z) * kMmaCols, m = col / n;
    const uint32_t q = sa.ra.q[m];
    const uint64_t mu = sa.mu[m];
    const uint32_t *vb = a.v + z * a.vstride + col + c;
    WideSum s[16];
    for (int i0 = 0; i0 < l; i0 += KS) {
      __syncthreads();
      for (int t = threadIdx.x; t < KS * kMmaKeys; t += kMmaThreads) {
        const int i = t % KS, k = t / KS;
        ystage[i * PITCH + k] =
            i0 + i < l && key0 + k < a.nkeys ? y_residue(a.y[(size_t)(key0 + k) * l + i0 + i], a.y_signed, q, mu) : 0u;
      }
      __syncthreads();
      for (int i = 0; i < KS; i += 4) {
        uint32_t x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = i0 + i + u < l ? __ldg(vb + (size_t)(i0 + i + u) * 3 * n) : 0u;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
#pragma unroll
          for (int u = 0; u < 4; u += 2) {
            const uint4 w0 = *reinterpret_cast<const uint4 *>(ystage + (i + u) * PITCH + kg * 16 + 4 * g);
            const uint4 w1 = *reinterpret_cast<const uint4 *>(ystage + (i + u + 1) * PITCH + kg * 16 + 4 * g);
            s[4 * g].add((uint64_t)x[u] * w0.x + (uint64_t)x[u + 1] * w1.x);
            s[4 * g + 1].add((uint64_t)x[u] * w0.y + (uint64_t)x[u + 1] * w1.y);
            s[4 * g + 2].add((uint64_t)x[u] * w0.z + (uint64_t)x[u + 1] * w1.z);
            s[4 * g + 3].add((uint64_t)x[u] * w0.w + (uint64_t)x[u + 1] * w1.w);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int key = key0 + kg * 16 + k;
      if (key < a.nkeys)
        a.out[(size_t)(z * (size_t)a.nkeys + key) * 3 * n + col + c] = s[k].mod(mu, q);
    }
  }
}

__global__ void __launch_bounds__(kMmaThreads, 1) 
    k_mac_mma(const __grid_constant__ MmaArgs a, const __grid_constant__ SchemeArgs sa, uint32_t *__restrict__ status) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int n = sa.ra.n, l = sa.l, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks = (l + kMmaK - 1) / kMmaK;
  const uint32_t smem_a = smem_u32_addr(smem);
  const uint32_t smem_b = smem_a + (uint32_t)chunks * (kMmaK / 16) * kMmaLboA;
  const uint32_t bars = smem_b + 2 * kMmaStage, slot = bars + 16;
  const int key0 = (blockIdx.x % a.key_tiles) * kMmaKeys;
  const int first = blockIdx.x / a.key_tiles, stride = gridDim.x / a.key_tiles;
  const int per_z = 3 * n / kMmaCols, tiles = a.nz * per_z;
  // v of a step: the 16 slots 32 i + 4 kq + j (i, j < 4) of its 128, one coefficient per thread;
  // tile and chunk of the next step to load advance with each call
  const int c = tid & (kMmaCols - 1), kq = tid / kMmaCols;
  const int steps = first < tiles ? (tiles - first + stride - 1) / stride * chunks : 0;
  int ld_tile = first, ld_ch = 0;
  const uint32_t row_words = 3u * (uint32_t)n;
  const auto load = [&](uint32_t (&r)[16]) {
    if (ld_tile >= tiles) return;
    const int z = ld_tile / per_z, i0 = ld_ch * kMmaK + 4 * kq;
    const uint32_t *p = a.v + z * a.vstride + (ld_tile - z * per_z) * kMmaCols;
    uint32_t at = (uint32_t)i0 * row_words + (uint32_t)c;  // l 3n < 2^32 words
    if ((ld_ch + 1) * kMmaK <= l) {
#pragma unroll
      for (int i = 0; i < 4; ++i, at += 32 * row_words)
#pragma unroll
        for (int j = 0; j < 4; ++j) r[4 * i + j] = __ldg(p + (at + (uint32_t)j * row_words));
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i, at += 32 * row_words)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          r[4 * i + j] = i0 + 32 * i + j < l ? __ldg(p + (at + (uint32_t)j * row_words)) : 0u;
    }
    if (++ld_ch == chunks) ld_ch = 0, ld_tile += stride;
  };
  uint32_t ra[16], rb[16];
  load(ra);
  load(rb);
  if (warp == 0) tmem_alloc(slot, kMmaTmem);
  if (tid == 0) {
    mbar_init(bars, 1);
    mbar_init(bars + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // pack y: 8 keys per warp, 128 slots of each at a time (32 loads in flight per thread)
  bool bad = false;
  constexpr int KW = kMmaKeys / (kMmaThreads / 32);
  for (int ch = 0; ch < chunks; ++ch) {
    uint32_t w[KW][4];
#pragma unroll
    for (int k = 0; k < KW; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int key = key0 + warp * KW + k, row = ch * kMmaK + 32 * i + lane;
        w[k][i] = key < a.nkeys && row < l ? __ldg(a.y + (size_t)key * l + row) : 0u;
      }
#pragma unroll
    for (int k = 0; k < KW; ++k) {
#pragma unroll
      for (int i = 0; i < 4; ++i) bad |= a.y_signed ? w[k][i] + 128u > 255u : w[k][i] > 127u;
      const uint32_t lo = __byte_perm(w[k][0], w[k][1], 0x0040), hi = __byte_perm(w[k][2], w[k][3], 0x0040);
      const uint32_t off =
          (uint32_t)(ch * (kMmaK / 16) + (lane >> 2)) * kMmaLboA + (uint32_t)(warp * KW + k) * 16 + (lane & 3) * 4;
      *reinterpret_cast<uint32_t *>(smem + off) = __byte_perm(lo, hi, 0x5410);
    }
  }
  umma_fence_before();
  bad = __syncthreads_or(bad);
  umma_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot));
  if (bad) {
    mac_tiles_general(a, sa, reinterpret_cast<uint32_t *>(smem + (smem_b - smem_a)), key0, first, stride, tiles);
  } else {
    bool live = true;
    int tile = first, ch = 0;
    const auto body = [&](int s, uint32_t (&r)[16]) {
      const uint32_t st = (uint32_t)s & 1u, stage = smem_b + st * kMmaStage, bar = bars + 8 * st;
      if (s >= 2 && live) live = mbar_wait(bar, ((uint32_t)(s >> 1) - 1u) & 1u);  // step s - 2 has read this stage
      {
        uint32_t o[4][4];  // [slot quad j][byte b]
#pragma unroll
        for (int j = 0; j < 4; ++j) byte_transpose(r[j], r[4 + j], r[8 + j], r[12 + j], o[j]);
        uint8_t *dst = smem + (stage - smem_a) + kq * kMmaLboB + c * 16;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          *reinterpret_cast<uint4 *>(dst + b * kMmaCols * 16) = make_uint4(o[0][b], o[1][b], o[2][b], o[3][b]);
      }
      load(r);
      smem_fence_async();
      umma_fence_before();
      __syncthreads();
      if (tid == 0) {
        umma_fence_after();
#pragma unroll
        for (int j = 0; j < kMmaK / 32; ++j)
          umma_i8(tmem, umma_smem_desc(smem_a + (uint32_t)(ch * (kMmaK / 16) + 2 * j) * kMmaLboA, kMmaLboA),
                  umma_smem_desc(stage + 2 * j * kMmaLboB, kMmaLboB), kMmaIdesc, ch > 0 || j > 0);
        umma_commit(bar);
      }
      if (++ch < chunks) return;
      ch = 0;
      // epilogue: the thread's key (TMEM lane) by 16 coefficients, 8 at a time
      if (live) live = mbar_wait(bar, (uint32_t)(s >> 1) & 1u);
      umma_fence_after();
      const int z = tile / per_z, col = (tile - z * per_z) * kMmaCols, m = col / n;
      tile += stride;
      const uint32_t q = sa.ra.q[m], mul = a.mul[m];
      const uint64_t off = a.off[m];
      const int sh = a.sh[m];
      // through the free stages, so that rows of 256 bytes are stored whole
      uint32_t *row = reinterpret_cast<uint32_t *>(smem + (smem_b - smem_a)) + ((warp & 3) * 32 + lane) * kMmaPitch +
                      (warp >> 2) * 16;
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        uint32_t d[4][8];
#pragma unroll
        for (int b = 0; b < 4; ++b)
          tmem_ld8(tmem + ((uint32_t)(warp & 3) << 21) + b * kMmaCols + (warp >> 2) * 16 + h, d[b]);
        tmem_wait_ld();
        uint32_t x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int64_t lo = (int64_t)(int32_t)d[1][e] * 256 + (int32_t)d[0][e];
          const int64_t hi = (int64_t)(int32_t)d[3][e] * 256 + (int32_t)d[2][e];
          const uint64_t v = (uint64_t)(hi * 65536 + lo) + off;
          const uint32_t qe = __umulhi((uint32_t)(v >> 20), mul) >> sh;
          x[e] = mod_red1((uint32_t)v - qe * q, q);
        }
        *reinterpret_cast<uint4 *>(row + h) = make_uint4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<uint4 *>(row + h + 4) = make_uint4(x[4], x[5], x[6], x[7]);
      }
      __syncthreads();
      const int c4 = (tid & 15) * 4;
      uint32_t *o = a.out + (size_t)(z * (size_t)a.nkeys + key0) * 3 * n + col + c4;
      const uint32_t *src = reinterpret_cast<const uint32_t *>(smem + (smem_b - smem_a)) + c4;
#pragma unroll
      for (int k = tid >> 4; k < kMmaKeys; k += kMmaThreads / 16)
        if (key0 + k < a.nkeys) store4(o + (size_t)k * 3 * n, *reinterpret_cast<const uint4 *>(src + k * kMmaPitch), a.vec);
      __syncthreads();
    };
    for (int s = 0; s < steps; s += 2) {
      body(s, ra);
      if (s + 1 < steps) body(s + 1, rb);
    }
    if (!live && lane == 0) atomicOr(status, kStatusMmaTimeout);
  }
  umma_fence_before();
  __syncthreads();
  if (warp == 0) {
    umma_fence_after();
    tmem_free(tmem, kMmaTmem);
  }
}

}  // namespace

// From this many keys on the tensor-core kernel is used; its time does not depend on their number up to
// 128.  us on a B200 (n, l: streamed with 1, 2, 3, 4, 8 keys | tensor cores with 3): 4096, 784: 16.7,
// 20.6, 29.6, 30.9, 49.4 | 26.8; 2048, 200: 9.0, 10.4, 14.4, 15.6, 18.6 | 8.6; 1024, 40: 6.1, 8.4,
// 12.4, 14.2, 14.5 | 7.5.
constexpr int kMmaMinKeys = 3;

int mac_launch(Ctx &c, const SchemeArgs &sa, const uint32_t *d_v, size_t vstride, int nz, const uint32_t *d_y,
               int y_signed, int nkeys, uint32_t *d_out, cudaStream_t s) {
  const int n = c.n, l = c.l;
  const int vec = ((reinterpret_cast<uintptr_t>(d_v) | reinterpret_cast<uintptr_t>(d_out)) & 15u) == 0 && vstride % 4 == 0;
  if (nkeys >= kMmaMinKeys && n >= kMmaCols && l <= kMmaMaxL) {
    MmaArgs a{d_v, vstride, d_y, y_signed, nkeys, nz, (nkeys + kMmaKeys - 1) / kMmaKeys, vec, d_out, {}};
    for (int j = 0; j < 3; ++j) {
      const uint64_t q = sa.ra.q[j];
      a.off[j] = ((1ull << 50) / q + 1) * q;
      while (((1ull << 53) << a.sh[j]) / q < (1ull << 32)) ++a.sh[j];
      a.mul[j] = (uint32_t)(((1ull << 52) << a.sh[j]) / q);
    }
    const long long tiles = (long long)nz * (3 * n / kMmaCols);
    const long long per_key_tile = std::max(1LL, std::min(tiles, (long long)c.num_sms / a.key_tiles));
    const uint32_t smem = mma_smem(l);
    CUFE_CUDA(cudaFuncSetAttribute(k_mac_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    note_launch(), k_mac_mma<<<(unsigned)(per_key_tile * a.key_tiles), kMmaThreads, smem, s>>>(a, sa, c.d_status);
    CUFE_CUDA(cudaGetLastError());
    return CUFE_OK;
  }
  const int kch = nkeys >= 3 ? 4 : nkeys;
  const int groups = (nkeys + kch - 1) / kch;
  // 1 KB of a row per CTA where that leaves 8 CTAs per SM, else 256 bytes
  int lanes = std::min(n / 4, 64);
  if ((long long)nz * groups * 3 * n / (4 * lanes) < 8LL * c.num_sms) lanes = std::min(lanes, 16);
  const dim3 grid((unsigned)(3 * n / (4 * lanes)), (unsigned)nz, (unsigned)groups);
  note_launch();
  if (kch == 1)
    k_mac_few<1><<<grid, kFewThreads, 0, s>>>(d_v, vstride, d_y, y_signed, nkeys, d_out, lanes, vec, sa);
  else if (kch == 2)
    k_mac_few<2><<<grid, kFewThreads, 0, s>>>(d_v, vstride, d_y, y_signed, nkeys, d_out, lanes, vec, sa);
  else
    k_mac_few<4><<<grid, kFewThreads, 0, s>>>(d_v, vstride, d_y, y_signed, nkeys, d_out, lanes, vec, sa);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

}  // namespace cufe

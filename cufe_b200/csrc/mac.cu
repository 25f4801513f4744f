// mac.cu -- the l-sums of key generation and decryption:
//   out[z][k][m][j] = sum_{i < l} y[k][i] v[z][i][m][j] mod q_m
// for keys k, RNS moduli m and coefficients j, with v = msk (src/rlwe_sife.c:215-245) or the
// ciphertexts z (the sum of src/rlwe_sife.c:248-278).
//
// Three kernels.  k_mac_few streams v once per KCH keys and is bound by memory; k_mac_mma is the
// product of many keys with v on the tensor cores; k_mac_short takes sums of a few rows.  Before, every product was three integer
// instructions and v was read once per 4 keys (key generation) or per key (decryption).  B200,
// us per call, before -> now: 1 key at n = 4096, l = 784 277 -> 13; 591 keys at l = 785 2034 -> 70;
// the decryption of one ciphertext under 591 keys at n = 2048, l = 124 254 -> 100 (60 with its transforms read
// where they lie and launched at once).
#include <algorithm>
#include <cmath>

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

// x mod q for |x| < 2^63
__device__ __forceinline__ uint32_t mod_s64(int64_t x, uint64_t mu, uint32_t q) {
  const uint32_t r = mod_u64((uint64_t)(x < 0 ? -x : x), mu, q);
  return x < 0 && r ? q - r : r;
}

// A CTA sums 4 * lanes coefficients of one (z, modulus) for KCH keys: thread (slice, lane) takes 4
// coefficients (16-byte loads) of the rows slice, slice + slices, ..., eight rows in flight, and
// the slices are added in shared memory, one thread per coefficient, so no partial sums go
// through memory.
struct FewArgs {
  const uint32_t *v, *y;
  size_t vstride;
  uint32_t *out;
  int y_signed, nkeys, lanes, vec;
};
template <int KCH>
struct FewSmem {
  uint32_t ys[KCH][kFewRows];
  uint64_t red[4 * kFewThreads];
  uint32_t redh[4 * kFewThreads];
};

// WIDE: 96-bit sums of the words by the residues of y.  Otherwise signed 64-bit sums, one
// multiply-add per product, for |y| < 2^15 (2^31 2^15 l <= 2^62) and words below 2^31; returns
// false, and stores nothing, where a word is not.  staged: the first rows of y are in sm.ys.
template <int KCH, bool WIDE>
__device__ __forceinline__ bool few_sums(const FewArgs &a, const SchemeArgs &sa, FewSmem<KCH> &sm, bool staged) {
  const int n = sa.ra.n, l = sa.l, tid = threadIdx.x, lanes = a.lanes;
  const int lane = tid & (lanes - 1), slice = tid / lanes, slices = kFewThreads / lanes;
  const int tiles = n / (4 * lanes);  // per residue polynomial
  const int m = blockIdx.x / tiles, j0 = 4 * (blockIdx.x - m * tiles) * lanes;
  const int z = blockIdx.y, k0 = blockIdx.z * KCH, keys = min(KCH, a.nkeys - k0);
  const uint32_t q = sa.ra.q[m];
  const uint64_t mu = sa.mu[m];
  const uint32_t *vb = a.v + z * a.vstride + (size_t)m * n + j0 + 4 * lane;
  const size_t row = (size_t)3 * n;
  uint64_t acc[KCH][4];
  uint32_t hi[KCH][4], any = 0;
#pragma unroll
  for (int kk = 0; kk < KCH; ++kk)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[kk][e] = 0, hi[kk][e] = 0;
  for (int r0 = 0; r0 < l; r0 += kFewRows) {
    const int rows = min(kFewRows, l - r0);
    if (r0 || !staged) {
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < KCH; ++kk)
        for (int i = tid; i < rows; i += kFewThreads) {
          const uint32_t w = kk < keys ? a.y[(size_t)(k0 + kk) * l + r0 + i] : 0u;
          sm.ys[kk][i] = WIDE ? y_residue(w, a.y_signed, q, mu) : w;
        }
      __syncthreads();
    }
    const uint32_t *vr = vb + (size_t)r0 * row;
    for (int i = slice; i < rows; i += 8 * slices) {
      uint4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = i + u * slices;
        x[u] = r < rows ? load4(vr + (size_t)r * row, a.vec) : make_uint4(0, 0, 0, 0);
      }
      if (!WIDE) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          any |= x[u].x | x[u].y | x[u].z | x[u].w;
#pragma unroll
          for (int kk = 0; kk < KCH; ++kk) {
            const int32_t yv = (int32_t)sm.ys[kk][min(i + u * slices, kFewRows - 1)];
            acc[kk][0] += (uint64_t)((int64_t)(int32_t)x[u].x * yv);
            acc[kk][1] += (uint64_t)((int64_t)(int32_t)x[u].y * yv);
            acc[kk][2] += (uint64_t)((int64_t)(int32_t)x[u].z * yv);
            acc[kk][3] += (uint64_t)((int64_t)(int32_t)x[u].w * yv);
          }
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < KCH; ++kk)
#pragma unroll
          for (int u = 0; u < 8; u += 2) {
            const uint32_t y0 = sm.ys[kk][min(i + u * slices, kFewRows - 1)];
            const uint32_t y1 = sm.ys[kk][min(i + (u + 1) * slices, kFewRows - 1)];
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
  if (!WIDE && __syncthreads_or((int32_t)any < 0)) return false;
  const int cols = 4 * lanes;
#pragma unroll
  for (int kk = 0; kk < KCH; ++kk) {
    if (kk >= keys) break;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sm.red[slice * cols + 4 * lane + e] = acc[kk][e];
      if (WIDE) sm.redh[slice * cols + 4 * lane + e] = hi[kk][e];
    }
    __syncthreads();
    uint32_t *o = a.out + ((size_t)(z * (size_t)a.nkeys + k0 + kk) * 3 + m) * n + j0;
    for (int i = tid; i < cols; i += kFewThreads) {
      if (WIDE) {
        WideSum w;
        for (int s = 0; s < slices; ++s) {
          w.add(sm.red[s * cols + i]);
          w.hi += sm.redh[s * cols + i];
        }
        o[i] = w.mod(mu, q);
      } else {
        uint64_t t = 0;
        for (int s = 0; s < slices; ++s) t += sm.red[s * cols + i];
        o[i] = mod_s64((int64_t)t, mu, q);
      }
    }
  }
  return true;
}

template <int KCH>
__global__ void __launch_bounds__(kFewThreads, KCH == 4 ? 2 : KCH == 2 ? 3 : 4)
    k_mac_few(const __grid_constant__ FewArgs a, const __grid_constant__ SchemeArgs sa) {
  __shared__ FewSmem<KCH> sm;
  const int l = sa.l, k0 = blockIdx.z * KCH, keys = min(KCH, a.nkeys - k0);
  // y of the first rows staged and checked at once, the rows beyond them checked
  bool big = false;
#pragma unroll
  for (int kk = 0; kk < KCH; ++kk)
    for (int i = threadIdx.x; i < l; i += kFewThreads) {
      const uint32_t w = kk < keys ? a.y[(size_t)(k0 + kk) * l + i] : 0u;
      if (i < kFewRows) sm.ys[kk][i] = w;
      big |= a.y_signed ? w + 32767u > 65534u : w > 32767u;
    }
  big = __syncthreads_or(big);
  if (!big && few_sums<KCH, false>(a, sa, sm, true)) return;
  few_sums<KCH, true>(a, sa, sm, false);
}

// ------------------------------------------------------------------ short sums

// A thread sums one coefficient for four keys over all rows: no slices to add up and no packing, so the
// shortest way through sums of a few rows, whatever the weights (Shoup products of their residues).
constexpr int kShortRows = 128, kShortKeys = 4;
__global__ void __launch_bounds__(256) k_mac_short(const __grid_constant__ FewArgs a, const __grid_constant__ SchemeArgs sa) {
  __shared__ uint2 ys[kShortKeys][kShortRows];  // (y, floor(y 2^32 / q))
  const int n = sa.ra.n, l = sa.l, z = blockIdx.y / 3, m = blockIdx.y - 3 * z, k0 = blockIdx.z * kShortKeys;
  const uint32_t q = sa.ra.q[m];
  const uint64_t mu = sa.mu[m];
  for (int t = threadIdx.x; t < kShortKeys * l; t += blockDim.x) {
    const int kk = t / l, i = t - kk * l;
    const uint32_t w = k0 + kk < a.nkeys ? y_residue(a.y[(size_t)(k0 + kk) * l + i], a.y_signed, q, mu) : 0u;
    const uint64_t ws = (uint64_t)w << 32, qe = __umul64hi(ws, mu);  // floor(ws / q) or one less
    ys[kk][i] = make_uint2(w, (uint32_t)qe + (uint32_t)(ws - qe * q >= q));
  }
  __syncthreads();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t *v = a.v + z * a.vstride + (size_t)m * n + j;
  uint64_t acc[kShortKeys] = {};
#pragma unroll 8
  for (int i = 0; i < l; ++i) {
    const uint32_t x = __ldg(v + (size_t)i * 3 * n);
#pragma unroll
    for (int kk = 0; kk < kShortKeys; ++kk) acc[kk] += shoup_lazy(x, ys[kk][i].x, ys[kk][i].y, q);
  }
  uint32_t *o = a.out + ((size_t)(z * (size_t)a.nkeys + k0) * 3 + m) * n + j;
#pragma unroll
  for (int kk = 0; kk < kShortKeys; ++kk)
    if (k0 + kk < a.nkeys) o[(size_t)kk * 3 * n] = mod_u64(acc[kk], mu, q);
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
  // Reduction of a sum s, |s| < 2^50 (l <= 1280), by recip20: with off a multiple of q of at least 2^50 and
  // below 2^50 + 2^31, s + off is in [0, 2^51 + 2^31)
  uint64_t off[3];
  uint32_t mul[3];
  int sh[3];
};

// The same tiles where a key has an entry outside a signed byte: Shoup products of the residues of y
// (three 32-bit multiplications; a 64-bit multiply-add takes as long as four), two coefficients and
// 8 keys per thread.  The 16 warps take the groups of 8 keys that hold keys, times slices of the
// rows, 16 of them at a time each; the slices' residues are added at the end.
__device__ __noinline__ void mac_tiles_general(const MmaArgs &a, const SchemeArgs &sa, uint8_t *smem, int key0,
                                               int first, int stride, int tiles) {
  constexpr int ROWS = 16, KT = 8, WARPS = kMmaThreads / 32, PER = ROWS * KT * WARPS / kMmaThreads;
  uint2 *ystage = reinterpret_cast<uint2 *>(smem);      // (y, floor(y 2^32 / q)) of [row][key]
  uint32_t *part = reinterpret_cast<uint32_t *>(smem);  // [slice][key][coefficient]
  const int n = sa.ra.n, l = sa.l, per_z = 3 * n / kMmaCols, tid = threadIdx.x;
  const int c = tid & 31, g = tid >> 5;
  const int live = min(kMmaKeys, a.nkeys - key0);
  int groups = 1;
  while (groups * KT < live) groups *= 2;
  const int slices = WARPS / groups, keys = KT * groups, pitch = keys + 2, rows = ROWS * slices;
  const int kg = g % groups, sl = g / groups;
  for (int tile = first; tile < tiles; tile += stride) {
    const int z = tile / per_z, col = (tile - z * per_z) * kMmaCols, m = col / n;
    const uint32_t q = sa.ra.q[m];
    const uint64_t mu = sa.mu[m];
    const uint32_t *vb = a.v + z * a.vstride + col + c;
    uint64_t s[KT][2];
#pragma unroll
    for (int k = 0; k < KT; ++k) s[k][0] = s[k][1] = 0;
    uint32_t yn[PER];  // the y of the next rows, loaded while these are multiplied
    const auto load_y = [&](int i0) {
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int t = tid + u * kMmaThreads, r = i0 + t % rows, k = t / rows;
        yn[u] = r < l && k < live ? __ldg(a.y + (size_t)(key0 + k) * l + r) : 0u;
      }
    };
    load_y(0);
    for (int i0 = 0; i0 < l; i0 += rows) {
      uint32_t x[ROWS][2];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int r = i0 + sl * ROWS + i;
        x[i][0] = r < l ? __ldg(vb + (size_t)r * 3 * n) : 0u;
        x[i][1] = r < l ? __ldg(vb + (size_t)r * 3 * n + 32) : 0u;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int t = tid + u * kMmaThreads, i = t % rows, k = t / rows;
        const uint32_t w = y_residue(yn[u], a.y_signed, q, mu);
        const uint64_t ws = (uint64_t)w << 32, qe = __umul64hi(ws, mu);  // floor(ws / q) or one less
        ystage[i * pitch + k] = make_uint2(w, (uint32_t)qe + (uint32_t)(ws - qe * q >= q));
      }
      __syncthreads();
      load_y(i0 + rows);
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int e = 0; e < KT; e += 2) {
          const uint4 w = *reinterpret_cast<const uint4 *>(ystage + (sl * ROWS + i) * pitch + kg * KT + e);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            s[e][h] += shoup_lazy(x[i][h], w.x, w.y, q);
            s[e + 1][h] += shoup_lazy(x[i][h], w.z, w.w, q);
          }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) part[(sl * keys + kg * KT + k) * kMmaCols + c + 32 * h] = mod_u64(s[k][h], mu, q);
    __syncthreads();
    for (int t = tid; t < live * kMmaCols; t += kMmaThreads) {
      uint64_t sum = 0;
      for (int u = 0; u < slices; ++u) sum += part[u * keys * kMmaCols + t];
      a.out[(size_t)(z * (size_t)a.nkeys + key0 + t / kMmaCols) * 3 * n + col + t % kMmaCols] = mod_u64(sum, mu, q);
    }
    __syncthreads();
  }
}
static_assert(16 * 16 * (8 + 2) * 8 <= 2 * kMmaStage && 16 * (128 + 2) * 8 <= 2 * kMmaStage &&
                  128 * kMmaCols * 4 <= 2 * kMmaStage,
              "the general tiles' staging");

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
    mac_tiles_general(a, sa, smem + (smem_b - smem_a), key0, first, stride, tiles);
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
      __syncwarp();  // thread 0's warp waits for the products only when they have been issued
      if (++ch < chunks) return;
      ch = 0;
      // epilogue: the thread's key (TMEM lane) by 16 coefficients, 8 at a time
      if (live) live = mbar_wait(bar, (uint32_t)(s >> 1) & 1u);
      __syncwarp();  // the wait's loop may leave a warp's threads apart, and the accumulator loads take whole warps
      umma_fence_after();
      const int z = tile / per_z, col = (tile - z * per_z) * kMmaCols, m = col / n;
      tile += stride;
      const uint32_t q = sa.ra.q[m], mul = a.mul[m];
      const uint64_t off = a.off[m];
      const int sh = a.sh[m];
      // through the free stages, so that rows of 256 bytes are stored whole
      uint32_t *row = reinterpret_cast<uint32_t *>(smem + (smem_b - smem_a)) + ((warp & 3) * 32 + lane) * kMmaPitch +
                      (warp >> 2) * 16;
      const bool any = key0 + (warp & 3) * 32 < a.nkeys;  // whole warps
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        if (!any) break;
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

// Coefficients / 4 of a streamed CTA.  About 64 rows or more per slice; fewer, and so more slices and CTAs, while
// there are not two CTAs per SM and, with three keys or more, whose slices cost more to add up, more than the eight rows that
// are in flight at once (1 key at n = 4096, l = 784: 12.5 us with 384 CTAs, 16.6 with 192; 3 keys at l = 8: 6 us in one slice, 10 in 32).
static int few_lanes(const Ctx &c, int nz, int keys, int groups) {
  int lanes = 256;
  while (lanes > 16 && c.l / (kFewThreads / lanes) >= 128) lanes /= 2;
  lanes = std::min(lanes, c.n / 4);
  while (lanes > 8 && (keys < 3 || c.l > 8 * (kFewThreads / lanes)) &&
         (long long)nz * groups * 3 * c.n / (4 * lanes) < 2LL * c.num_sms)
    lanes /= 2;
  return lanes;
}

// Which kernel, of three keys or more (fewer are streamed): the least of these estimates, us on a B200.
//   streamed: waves of two CTAs per SM, each 5 to 7.5 by its columns and 1.6 per further 8 rows of a slice; and v read at
//     3.5 TB/s per 4 keys;
//   tensor cores: the CTAs walk their coefficient tiles, 1.25 per 128 slots and 1.5 per epilogue, whatever
//     the number of keys up to 128 per tile;
//   short: 2.85 M products a us behind a latency of the rows; below 32 rows, and in rings below 64.
// us measured (streamed | tensor cores | short) at n, l, ciphertexts, keys: 4096, 37, 21, 3: 21 | 78; 2048, 53,
// 26, 3: 22 | 52; 4096, 123, 36, 4: 70 | 127; 4096, 65, 17, 8: 43 | 66; 4096, 784, 4, 4: 60 | 65; 4096, 100, 8, 16:
// 54 | 36; 4096, 784, 1, 8: 30 | 24; 4096, 100, 1, 12: 11 | 9; 4096, 32, 1, 8: 6 | 9; 1024, 100, 1, 32: 10 | 6; 1024,
// 8, 1, 16: 7 | 6 | 4; 4096, 8, 1, 16: 7 | 9 | 4; 4096, 16, 1, 64: 12 | 9 | 10; 4096, 8, 1, 600: 46 | 25 | 42.
enum MacKernel { kMacFew, kMacMma, kMacShort };
static MacKernel choose_kernel(const Ctx &c, int nz, int nkeys) {
  if (nkeys < 2) return kMacFew;
  const int groups = (nkeys + 3) / 4, lanes = few_lanes(c, nz, nkeys, groups), slices = kFewThreads / lanes;
  const double ctas = (double)nz * groups * 3 * c.n / (4 * lanes), waves = ctas / (2 * c.num_sms);
  const double per_wave = 5.0 + 2.5 * lanes / 256 + 1.6 * (((c.l + slices - 1) / slices + 7) / 8 - 1);
  double best = std::max(0.8 + (waves < 4 ? std::ceil(waves) : waves) * per_wave,
                         5.0 + (double)groups * nz * c.l * 12.0 * c.n / 3.5e6);
  MacKernel kernel = kMacFew;
  if (nkeys == 2) best = 4.6;  // streamed in short sums; never on the tensor cores
  if (nkeys > 2 && c.n >= kMmaCols && c.l <= kMmaMaxL) {
    const int key_tiles = (nkeys + kMmaKeys - 1) / kMmaKeys;
    const long long tiles = (long long)nz * (3 * c.n / kMmaCols);
    const long long each = std::max(1LL, (long long)c.num_sms / key_tiles), rounds = (tiles + each - 1) / each;
    const double us = 4.0 + (double)rounds * (1.25 * ((c.l + kMmaK - 1) / kMmaK) + 1.5);
    if (us < best) best = us, kernel = kMacMma;
  }
  if ((c.l < 32 || (c.n < kMmaCols && c.l <= kShortRows)) && nz <= 21845 && groups < 65536 &&
      2.5 + 0.16 * c.l + (double)nz * groups * 12.0 * c.n * (c.l + 7) / 2.85e6 < best)
    kernel = kMacShort;
  return kernel;
}

int mac_launch(Ctx &c, const SchemeArgs &sa, const uint32_t *d_v, size_t vstride, int nz, const uint32_t *d_y,
               int y_signed, int nkeys, uint32_t *d_out, cudaStream_t s) {
  const int n = c.n, l = c.l;
  const int vec = ((reinterpret_cast<uintptr_t>(d_v) | reinterpret_cast<uintptr_t>(d_out)) & 15u) == 0 && vstride % 4 == 0;
  const MacKernel kernel = choose_kernel(c, nz, nkeys);
  if (kernel == kMacShort) {
    const FewArgs a{d_v, d_y, vstride, d_out, y_signed, nkeys, 0, 0};
    note_launch(), k_mac_short<<<dim3((n + 255) / 256, 3u * nz, (nkeys + kShortKeys - 1) / kShortKeys), 256, 0, s>>>(a, sa);
    CUFE_CUDA(cudaGetLastError());
    return CUFE_OK;
  }
  if (kernel == kMacMma) {
    MmaArgs a{d_v, vstride, d_y, y_signed, nkeys, nz, (nkeys + kMmaKeys - 1) / kMmaKeys, vec, d_out, {}};
    for (int j = 0; j < 3; ++j) {
      const uint64_t q = sa.ra.q[j];
      a.off[j] = ((1ull << 50) / q + 1) * q;
      a.mul[j] = recip20(q).mul;
      a.sh[j] = recip20(q).sh;
    }
    const long long tiles = (long long)nz * (3 * n / kMmaCols);
    const long long per_key_tile = std::max(1LL, std::min(tiles, (long long)c.num_sms / a.key_tiles));
    const uint32_t smem = mma_smem(l);
    // the limit of the longest l whatever this one: the attribute is the kernel's, and another context's thread may
    // set it between here and the launch
    CUFE_CUDA(cudaFuncSetAttribute(k_mac_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mma_smem(kMmaMaxL)));
    note_launch(), k_mac_mma<<<(unsigned)(per_key_tile * a.key_tiles), kMmaThreads, smem, s>>>(a, sa, c.d_status);
    CUFE_CUDA(cudaGetLastError());
    return CUFE_OK;
  }
  const int kch = nkeys >= 3 ? 4 : nkeys;
  const int groups = (nkeys + kch - 1) / kch;
  const int lanes = few_lanes(c, nz, nkeys, groups);
  const dim3 grid((unsigned)(3 * n / (4 * lanes)), (unsigned)nz, (unsigned)groups);
  const FewArgs a{d_v, d_y, vstride, d_out, y_signed, nkeys, lanes, vec};
  note_launch();
  if (kch == 1)
    k_mac_few<1><<<grid, kFewThreads, 0, s>>>(a, sa);
  else if (kch == 2)
    k_mac_few<2><<<grid, kFewThreads, 0, s>>>(a, sa);
  else
    k_mac_few<4><<<grid, kFewThreads, 0, s>>>(a, sa);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

}  // namespace cufe

// coef0.cu -- constant-coefficient decryption of many (ciphertext, key) pairs on the tensor cores.
//
// Per modulus m the residues are a product over K = n + l slots (see k_dec_coef0_tiled in ipfe.cu):
//   d0[c][k][m] = sum_{t < n} c_l[t] b_t + sum_{i < l} c_i[0] y_i,  b_0 = -s[0], b_t = s[n - t].
// Both factors are 31-bit residues, so each is taken as four unsigned bytes: byte a of the
// ciphertext times byte b of the key adds to the diagonal a + b of the result.  A: four byte planes of
// 128 ciphertexts; B: one operand of 256 rows, byte b of 64 keys at row 64 b + key.  The product of
// plane a with B then covers the four diagonals a .. a + 3, which lie side by side in TMEM, 64
// columns each, so one instruction per plane accumulates them all.  A diagonal is at most
// 4 * 255^2 * K < 2^31 for K <= 8192.  The epilogue puts the seven diagonals together mod q.
//
// k_coef0_pack writes both operands once as byte planes in the tensor core's shared-memory layout, in
// blocks of 64 slots, and k_coef0_mma streams the blocks of its tile with bulk copies.  Staged by
// the product kernel itself, every ciphertext was transposed once per 64 keys, and its c_i[0], one
// word per 12 n bytes, gathered as often.  The K range is split over CTAs where the tiles alone
// leave SMs idle; k_coef0_finish adds the parts and decodes.  1,000 ciphertexts x 500 keys at n = 2048,
// l = 124 on a B200, us: integer-pipe tiles 1,188; staged in the kernel 161; packed 88
// (23 pack, 52 product, 9 finish).
#include <algorithm>

#include "ctx.h"
#include "prof.h"
#include "scheme.cuh"
#include "umma.cuh"

namespace cufe {

namespace {

constexpr int kC0Threads = 256, kC0Cts = 128, kC0Keys = 64, kC0Slots = 64;
constexpr uint32_t kC0LboA = kC0Cts * 16, kC0LboB = 4 * kC0Keys * 16;
constexpr uint32_t kC0PlaneA = kC0Slots / 16 * kC0LboA;
constexpr uint32_t kC0BlockA = 4 * kC0PlaneA, kC0BlockB = kC0Slots / 16 * kC0LboB;  // 32 and 16 KB
constexpr uint32_t kC0StageBytes = kC0BlockA + kC0BlockB;
constexpr int kC0Stages = 4;
constexpr uint32_t kC0Smem = kC0Stages * kC0StageBytes + 128;
constexpr uint32_t kC0Tmem = 512;
constexpr uint32_t kC0Idesc = umma_i8_desc(false, 4 * kC0Keys);
constexpr int kC0Pitch = kC0Keys + 1;  // words per ciphertext of the staged output
static_assert(kC0Cts * kC0Pitch * 4 <= kC0Stages * kC0StageBytes, "the output fits the stages");

struct Coef0Args {
  const uint32_t *ct, *y, *sky;
  int y_signed, nct, nkeys, vec;
  int ct_tiles, key_tiles, chunks, poly_chunks, splits;
  uint8_t *pa, *pb;  // packed blocks [tile][m][chunk]
  uint32_t *part;    // [split][m][pair]
  uint32_t mul[3];  // recip20
  int sh[3];
};

// One thread: 16 consecutive slots of one row (a ciphertext, or a key) and modulus, as 16 bytes of
// each byte plane.  The four threads of a row read 256 contiguous bytes of c_l or s; 8 rows make
// 128-byte runs of the packed planes.
__global__ void __launch_bounds__(256) k_coef0_pack(const __grid_constant__ Coef0Args a, const __grid_constant__ SchemeArgs sa) {
  const int n = sa.ra.n, l = sa.l;
  const int k16 = threadIdx.x & 3, chunk = blockIdx.y, m = blockIdx.z;
  const long long row = (long long)blockIdx.x * 64 + (threadIdx.x >> 2);
  const long long ct_rows = (long long)a.ct_tiles * kC0Cts;
  uint32_t w[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) w[e] = 0;
  const int t = chunk * kC0Slots + 16 * k16, u = t - n;  // slot of the polynomial part, or of the l part
  uint8_t *dst;
  uint32_t plane;  // byte distance of two planes
  if (row < ct_rows) {
    if (row < a.nct) {
      const uint32_t *cb = a.ct + (size_t)row * (l + 1) * 3 * n + (size_t)m * n;
      if (chunk < a.poly_chunks) {
        const uint32_t *p = cb + (size_t)l * 3 * n + t;
        if (a.vec) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + i);
            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) w[e] = __ldg(p + e);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (u + e < l) w[e] = __ldg(cb + (size_t)(u + e) * 3 * n);
      }
    }
    dst = a.pa + ((size_t)(row / kC0Cts * 3 + m) * a.chunks + chunk) * kC0BlockA + k16 * kC0LboA + (row % kC0Cts) * 16;
    plane = kC0PlaneA;
  } else {
    const long long key = row - ct_rows;
    if (key >= (long long)a.key_tiles * kC0Keys) return;
    if (key < a.nkeys) {
      const uint32_t q = sa.ra.q[m];
      if (chunk < a.poly_chunks) {  // s[n - t], s[n - t - 1], ..: the 16 words below s[n - t], and that word
        const uint32_t *s = a.sky + ((size_t)key * 3 + m) * n;
        const uint32_t first = __ldg(s + (t ? n - t : 0));
        const uint32_t *p = s + n - t - 16;
        uint32_t v[16];
        if (a.vec) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 x = __ldg(reinterpret_cast<const uint4 *>(p) + i);
            v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = __ldg(p + e);
        }
        w[0] = t ? first : (first ? q - first : 0u);
#pragma unroll
        for (int e = 1; e < 16; ++e) w[e] = v[16 - e];
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (u + e < l) w[e] = y_residue(__ldg(a.y + (size_t)key * l + u + e), a.y_signed, q, sa.mu[m]);
      }
    }
    dst = a.pb + ((size_t)(key / kC0Keys * 3 + m) * a.chunks + chunk) * kC0BlockB + k16 * kC0LboB + (key % kC0Keys) * 16;
    plane = kC0Keys * 16;
  }
  uint32_t o[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) byte_transpose(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3], o[i]);
#pragma unroll
  for (int b = 0; b < 4; ++b)
    *reinterpret_cast<uint4 *>(dst + b * plane) = make_uint4(o[0][b], o[1][b], o[2][b], o[3][b]);
}

__global__ void __launch_bounds__(kC0Threads, 1)
    k_coef0_mma(const __grid_constant__ Coef0Args a, const __grid_constant__ SchemeArgs sa, uint32_t *__restrict__ status) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m = blockIdx.z % 3, split = blockIdx.z / 3;
  const uint32_t q = sa.ra.q[m];
  const uint32_t stage0 = smem_u32_addr(smem), bars = stage0 + kC0Stages * kC0StageBytes;
  const uint32_t full = bars, empty = bars + 8 * kC0Stages, done = empty + 8 * kC0Stages, slot = done + 8;
  const int ch0 = (int)((long long)a.chunks * split / a.splits), ch1 = (int)((long long)a.chunks * (split + 1) / a.splits);
  if (warp == 0) tmem_alloc(slot, kC0Tmem);
  if (tid == 0) {
    for (int i = 0; i < 2 * kC0Stages + 1; ++i) mbar_init(bars + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot));
  // this warp's TMEM lanes; it zeroes and later reads half of their columns
  const uint32_t quarter = tmem + ((uint32_t)(warp & 3) << 21);
  bool live = true;
  // warp 2's first thread copies: the first stages before the CTA's barrier, the others after it (they
  // wait for products, which are issued after it)
  const auto copy = [&](int ch) {
    const int st = (ch - ch0) % kC0Stages;
    const uint32_t stage = stage0 + st * kC0StageBytes;
    mbar_expect(full + 8 * st, kC0StageBytes);
    bulk_load(stage, a.pa + ((size_t)(blockIdx.x * 3 + m) * a.chunks + ch) * kC0BlockA, kC0BlockA, full + 8 * st);
    bulk_load(stage + kC0BlockA, a.pb + ((size_t)(blockIdx.y * 3 + m) * a.chunks + ch) * kC0BlockB, kC0BlockB,
              full + 8 * st);
  };
  if (tid == 64)
    for (int ch = ch0; ch < min(ch1, ch0 + kC0Stages); ++ch) copy(ch);
  __syncwarp();
  for (int i = 0; i < 7 * kC0Keys / 16; ++i) tmem_zero8(quarter + (uint32_t)((warp >> 2) * 7 * kC0Keys / 2 + 8 * i));
  tmem_wait_st();
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  if (tid == 64)
    for (int ch = ch0 + kC0Stages; ch < ch1 && live; ++ch) {
      live = mbar_wait(empty + 8 * ((ch - ch0) % kC0Stages), (uint32_t)((ch - ch0) / kC0Stages - 1) & 1u);
      if (live) copy(ch);
    }
  if (tid == 32) {  // warp 1's first thread issues the products
    for (int ch = ch0; ch < ch1 && live; ++ch) {
      const int s = ch - ch0, st = s % kC0Stages;
      live = mbar_wait(full + 8 * st, (uint32_t)(s / kC0Stages) & 1u);
      if (!live) break;
      umma_fence_after();
      const uint32_t stage = stage0 + st * kC0StageBytes;
#pragma unroll
      for (int j = 0; j < kC0Slots / 32; ++j)
#pragma unroll
        for (int p = 0; p < 4; ++p)
          umma_i8(tmem + p * kC0Keys, umma_smem_desc(stage + p * kC0PlaneA + 2 * j * kC0LboA, kC0LboA),
                  umma_smem_desc(stage + kC0BlockA + 2 * j * kC0LboB, kC0LboB), kC0Idesc, true);
      umma_commit(empty + 8 * st);
    }
    umma_commit(done);  // covers every product so far
  }
  __syncwarp();
  live = mbar_wait(done, 0) && live;
  if (!live) atomicOr(status, kStatusMmaTimeout);
  umma_fence_after();
  __syncthreads();  // every copy has been consumed: the stages hold the output now
  uint32_t *row = reinterpret_cast<uint32_t *>(smem) + ((warp & 3) * 32 + lane) * kC0Pitch + (warp >> 2) * 32;
  const uint32_t mul = a.mul[m];
  const int sh = a.sh[m];
  const auto reduce = [&](uint64_t x) {
    return mod_red1((uint32_t)x - (__umulhi((uint32_t)(x >> 20), mul) >> sh) * q, q);
  };
#pragma unroll 1
  for (int h = 0; h < 32; h += 8) {
    uint32_t d[7][8];
#pragma unroll
    for (int g = 0; g < 7; ++g) tmem_ld8(quarter + g * kC0Keys + (warp >> 2) * 32 + h, d[g]);
    tmem_wait_ld();
#pragma unroll
    for (int e = 0; e < 8; ++e) {  // Horner in steps of 2^16; every argument is below 2^48
      const auto two = [&](int g) { return (uint64_t)d[g + 1][e] * 256 + d[g][e]; };
      uint32_t r = reduce((uint64_t)d[6][e] * 65536 + two(4));
      r = reduce((uint64_t)r * 65536 + two(2));
      row[h + e] = reduce((uint64_t)r * 65536 + two(0));
    }
  }
  umma_fence_before();
  __syncthreads();
  if (warp == 0) {
    umma_fence_after();
    tmem_free(tmem, kC0Tmem);
  }
  const int ct0 = blockIdx.x * kC0Cts, key0 = blockIdx.y * kC0Keys;
  uint32_t *out = a.part + ((size_t)split * 3 + m) * a.nct * a.nkeys;
  for (int i = tid; i < kC0Cts * kC0Keys; i += kC0Threads) {
    const int c = i / kC0Keys, k = i % kC0Keys;
    if (ct0 + c < a.nct && key0 + k < a.nkeys)
      out[(size_t)(ct0 + c) * a.nkeys + key0 + k] = reinterpret_cast<const uint32_t *>(smem)[c * kC0Pitch + k];
  }
}

// adds the splits of every pair and decodes it
__global__ void __launch_bounds__(256) k_coef0_finish(const uint32_t *__restrict__ part, int splits, long long npairs,
                                                      uint32_t *__restrict__ out, DecodeArgs d) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npairs) return;
  uint32_t r0 = 0, r1 = 0, r2 = 0;
  for (int s = 0; s < splits; ++s) {
    const uint32_t *v = part + (size_t)s * 3 * npairs + p;
    r0 = mod_add(r0, v[0], d.q0);
    r1 = mod_add(r1, v[npairs], d.q1);
    r2 = mod_add(r2, v[2 * npairs], d.q2);
  }
  out[p] = decode_one(r0, r1, r2, d);
}

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

struct Coef0Plan {
  int ct_tiles, key_tiles, chunks, poly_chunks, splits;
  size_t pa, pb, part;  // bytes
};

// Splits of the K range: the number (up to 16, at least a chunk each) with the least estimated time,
// rounds of CTAs x (chunks of a CTA + its start and epilogue, about as long as 8 chunks).
Coef0Plan plan(const Ctx &c, int nct, int nkeys) {
  Coef0Plan p;
  p.ct_tiles = (nct + kC0Cts - 1) / kC0Cts;
  p.key_tiles = (nkeys + kC0Keys - 1) / kC0Keys;
  p.poly_chunks = c.n / kC0Slots;
  p.chunks = p.poly_chunks + (c.l + kC0Slots - 1) / kC0Slots;
  const long long tiles = (long long)p.ct_tiles * p.key_tiles * 3;
  p.splits = 1;
  double best = 1e30;
  for (int s = 1; s <= std::min(p.chunks, 16); ++s) {
    const double t = (double)((tiles * s + c.num_sms - 1) / c.num_sms) * ((double)p.chunks / s + 8.0);
    if (t < best * 0.97) best = t, p.splits = s;
  }
  p.pa = a256((size_t)p.ct_tiles * 3 * p.chunks * kC0BlockA);
  p.pb = a256((size_t)p.key_tiles * 3 * p.chunks * kC0BlockB);
  p.part = a256((size_t)p.splits * 3 * nct * nkeys * 4);
  return p;
}

}  // namespace

bool coef0_mma_ok(const Ctx &c) { return c.n >= kC0Slots && c.n + c.l <= 8192; }

size_t coef0_mma_bytes(const Ctx &c, int nct, int nkeys) {
  const Coef0Plan p = plan(c, nct, nkeys);
  return p.pa + p.pb + p.part;
}

int coef0_mma_slice(const Ctx &c, int nct, int nkeys, size_t bytes) {
  int m = nct;
  while (m > kC0Cts && coef0_mma_bytes(c, m, nkeys) > bytes) m = (m / 2 + kC0Cts - 1) / kC0Cts * kC0Cts;
  return m;
}

int coef0_mma_launch(Ctx &c, const SchemeArgs &sa, const DecodeArgs &dd, int nct, const uint32_t *d_ct, int nkeys,
                     const uint32_t *d_y, int y_signed, const uint32_t *d_sky, void *ws, uint32_t *d_out, cudaStream_t s) {
  const Coef0Plan p = plan(c, nct, nkeys);
  const long long npairs = (long long)nct * nkeys;
  Coef0Args a;
  a.ct = d_ct;
  a.y = d_y;
  a.sky = d_sky;
  a.y_signed = y_signed;
  a.nct = nct;
  a.nkeys = nkeys;
  a.vec = ((reinterpret_cast<uintptr_t>(d_ct) | reinterpret_cast<uintptr_t>(d_sky)) & 15u) == 0;
  a.ct_tiles = p.ct_tiles;
  a.key_tiles = p.key_tiles;
  a.chunks = p.chunks;
  a.poly_chunks = p.poly_chunks;
  a.splits = p.splits;
  a.pa = static_cast<uint8_t *>(ws);
  a.pb = a.pa + p.pa;
  a.part = reinterpret_cast<uint32_t *>(a.pb + p.pb);
  for (int j = 0; j < 3; ++j) {
    a.mul[j] = recip20(sa.ra.q[j]).mul;
    a.sh[j] = recip20(sa.ra.q[j]).sh;
  }
  CUFE_CUDA(cudaFuncSetAttribute(k_coef0_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kC0Smem));
  const unsigned rows = (unsigned)p.ct_tiles * kC0Cts + (unsigned)p.key_tiles * kC0Keys;
  note_launch(), k_coef0_pack<<<dim3(rows / 64, (unsigned)p.chunks, 3), 256, 0, s>>>(a, sa);
  CUFE_CUDA(cudaGetLastError());
  const dim3 grid((unsigned)p.ct_tiles, (unsigned)p.key_tiles, 3u * p.splits);
  note_launch(), k_coef0_mma<<<grid, kC0Threads, kC0Smem, s>>>(a, sa, c.d_status);
  CUFE_CUDA(cudaGetLastError());
  note_launch(), k_coef0_finish<<<(unsigned)((npairs + 255) / 256), 256, 0, s>>>(a.part, p.splits, npairs, d_out, dd);
  CUFE_CUDA(cudaGetLastError());
  return CUFE_OK;
}

}  // namespace cufe

// sampler_host.h -- host entry points of the sampler kernels (sampler.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstddef>

namespace cufe {

// the params.h RNS primes q_j = 2^k1 - 2^k2 + 1 (src/params.h:19)
constexpr uint32_t kRefPrimes[3] = {16760833u, 2147352577u, 2130706433u};

void aes_sbox(uint8_t out[256]);
// FIPS-197 key expansion into 60 big-endian round-key words
void aes_key_expand(const uint8_t key[32], uint32_t w[60]);

int sampler_init_device();
// device key expansion: d_rk[i][60] = aes_key_expand(d_seeds[d_perm ? d_perm[i] : i])
int expand_keys_device(const uint8_t *d_seeds, const uint32_t *d_perm, uint32_t count, uint32_t *d_rk,
                       cudaStream_t s);

// the parts of a CPU-mapping run, which may be launched by two calls: the candidates (num_sms CTAs
// at most), and the rest
enum { kSampleCandidates = 1, kSampleRest = 2, kSampleAll = 3 };
constexpr int kCandThreads = 512;  // threads of a candidate CTA, one CTA per SM

uint32_t cpu_map_refills(uint32_t calls, uint32_t n, int sig);

// Segmented form: S CPU-mapping streams of different lengths.  Stream s runs calls[s]
// sampler calls of n[s] samples; its refills occupy [roff[s], roff[s+1]) of the flattened
// refill space (multiples of 32), its call starts call_start[coff[s] + s .. coff[s+1] + s] (calls + 1
// entries), and the scatter writes its residues to out[ooff[s] + c * 3 n[s] ...][3][n[s]].  Round
// keys rkeys[s][60].  Without tables (n == nullptr) the streams are equal: u_calls calls of u_n
// samples, u_refills refills, output u_ostride words apart (mod 2^64: backwards too).
struct SegDev {
  uint32_t nstreams;
  const uint32_t *n, *calls;
  const uint64_t *roff, *coff, *ooff;
  uint32_t u_n, u_calls, u_refills;
  uint64_t u_ostride;
};
// How a run finds where its calls start (sampler.cu)
enum CallSearch : uint32_t { kSearchWalk, kSearchDoubling, kSearchTable };
struct SegSizes {
  uint32_t nstreams;
  uint64_t refills;
  uint64_t calls;
  uint32_t max_refills, max_calls, min_n;  // over the streams
  CallSearch search;
  uint32_t end_w;     // words per call of the table of call ends (kSearchTable)
  uint32_t end_mean;  // its windows follow this many times the mean overshoot: 1, or 0 or 2 to lead them astray
};
// another search for a run, before its scratch is laid out; false, and no change, where its sizes do not allow
// it (the walk they always do)
bool seg_search(SegSizes &z, CallSearch how);
// cufe_sampler_call_search: 0 the quickest, 1 the walk, 2 doubling where it is possible, for the sizes computed
// from now on
void set_call_search(int mode);
struct SegLayout {
  size_t n, calls, roff, coff, ooff, bytes;
};
// the tables of S streams in one buffer (device or host, same layout)
SegLayout seg_layout(uint32_t S);
SegDev seg_bind(void *base, uint32_t S);
// host: fill the tables (refills per stream from cpu_map_refills) into a host buffer of
// seg_layout(S).bytes; ooff may be NULL (candidates only)
SegSizes seg_fill_host(int sig, uint32_t S, const uint32_t *calls, const uint32_t *n, const uint64_t *ooff,
                       void *host_base);
size_t seg_scratch_bytes(const SegSizes &z);

// segmented run: candidates, scan, call starts and the scatter of the residues to d_out
int sample_cpu_map_seg(int sig, const SegDev &sg, const SegSizes &z, const uint32_t *d_rkeys, uint32_t *d_out,
                       void *scratch, uint32_t *d_status, int num_sms, cudaStream_t s, int parts = kSampleAll);

// CPU stream mapping: equal independent AES-CTR streams (round keys d_rkeys[nstreams][60], nonce 0, counter
// 0), each running `calls` consecutive sampler calls of n samples with sigma index sig; z from cpu_map_sizes,
// scratch of seg_scratch_bytes(z); residues written to d_out[nstreams][calls][3][n], those of the second of two
// streams to d_out1 where given.
SegSizes cpu_map_sizes(uint32_t nstreams, uint32_t calls, uint32_t n, int sig);
int sample_cpu_map(int sig, const SegSizes &z, const uint32_t *d_rkeys, uint32_t *d_out, void *ws, uint32_t *d_status,
                   int num_sms, cudaStream_t s, uint32_t *d_out1 = nullptr, int parts = kSampleAll);

// GPU counter mapping: polynomials poly0 .. poly0+npolys-1 of one key, residues to
// d_out[npolys][3][n].
int sample_gpu_map(int sig, const uint32_t *d_rkey, uint32_t poly0, uint32_t npolys, uint32_t n,
                   uint32_t *d_out, uint32_t *d_status, int num_sms, cudaStream_t s);

// uniform a (sample_polya): d_a[3][n]
int sample_polya(const uint32_t *d_rkey, uint32_t n, uint32_t *d_a, uint32_t *d_status, cudaStream_t s);

}  // namespace cufe

// M31 multilinear sum-check prover on the device (M31MultilinearSumcheckProofBuilderV1,
// SumcheckOracle.swift:797-868; statement digest :743-754; word digest :1288-1299;
// transcript frames :1066-1106).
//
// A table is proved by one group of warps: one warp computes the statement's word
// digest, a sequential sponge over the whole table (about 30,000 dependent
// permutations for 2^20 words), while the group's other warps sum the table for
// round 0; then the group proves the rounds.  A table of 2^20 words is 4 MiB, so
// each round is a few microseconds of one SM, and keeping a table in one group
// needs no grid-wide wait.  The single-table kernel is one CTA of 8 warps; the
// batched kernel packs four tables into one CTA (sumcheck_packed_kernel).
#include "azk_field.cuh"
#include "azk_internal.h"
#include "azk_transcript_warp.cuh"

namespace azk {

// Byte k of the framed word-digest input: u32 len || "AppleZKProver.M31Sumcheck.Words.V1"
// || u32 1 || u64 count || words (little-endian) (SumcheckOracle.swift:1288-1299).
__device__ __forceinline__ uint32_t digest_stream_byte(const uint32_t* words, uint64_t count, uint64_t k) {
  const char dom[] = "AppleZKProver.M31Sumcheck.Words.V1";
  if (k < 4) return (34u >> (8 * k)) & 0xFFu;
  if (k < 38) return (uint8_t)dom[k - 4];
  if (k < 42) return (1u >> (8 * (k - 38))) & 0xFFu;
  if (k < 50) return (uint32_t)(count >> (8 * (k - 42))) & 0xFFu;
  const uint64_t w = (k - 50) >> 2;
  return (__ldg(words + w) >> (8 * ((k - 50) & 3))) & 0xFFu;
}

// Rate word `lane` (< 17) of the block starting at stream byte `pos` >= 136 when
// the block lies inside the stream: after the 50-byte header every 8-byte word
// starts 2 bytes into a table word, so it is assembled from three table words.
// The three words are loaded before a permutation and assembled after it, so the
// load latency hides behind the permutation instead of stalling before it.
struct BlockWords {
  uint32_t w0 = 0, w1 = 0, w2 = 0;
  __device__ __forceinline__ void load(const uint32_t* words, uint64_t pos, uint32_t lane) {
    const uint32_t* w = words + ((pos - 50) >> 2) + 2 * lane;
    w0 = __ldg(w);
    w1 = __ldg(w + 1);
    w2 = __ldg(w + 2);
  }
  __device__ __forceinline__ uint64_t word() const { return ((uint64_t)w0 >> 16) | ((uint64_t)w1 << 16) | ((uint64_t)w2 << 48); }
};

// SHA3-256 of the framed table, by the whole warp (`col`: its 64-word shared
// exchange array, 16-byte aligned); lanes 0..3 return the digest lanes.
__device__ uint64_t digest_words_warp(const uint32_t* words, uint64_t count, uint64_t* col) {
  const uint32_t lane = threadIdx.x & 31;
  const WarpKeccak kf(lane, col);
  const uint64_t total = 50 + 4 * count;
  uint64_t a = 0;
  uint64_t pos = 0;
  if (total >= 136) {
    // first block: header bytes then table bytes
    if (lane < 17) {
      uint64_t v = 0;
      for (uint32_t b = 0; b < 8; b++) v |= (uint64_t)digest_stream_byte(words, count, 8 * lane + b) << (8 * b);
      a ^= v;
    }
    pos = 136;
    // full middle blocks, the next block's words loaded before this permutation
    BlockWords next;
    if (lane < 17 && pos + 136 <= total) next.load(words, pos, lane);
    kf.permute(a);
    while (pos + 136 <= total) {
      a ^= next.word();
      const uint64_t npos = pos + 136;
      next = BlockWords();
      if (lane < 17 && npos + 136 <= total) next.load(words, npos, lane);
      kf.permute(a);
      pos = npos;
    }
  }
  // final block: tail bytes, suffix 0x06, 0x80 at the end of the rate
  const uint64_t tail = total - pos;
  if (lane < 17) {
    uint64_t v = 0;
    for (uint32_t b = 0; b < 8; b++) {
      const uint64_t k = 8 * lane + b;
      if (k < tail) v |= (uint64_t)digest_stream_byte(words, count, pos + k) << (8 * b);
      if (k == tail) v |= (uint64_t)0x06 << (8 * b);
    }
    if (lane == 16) v ^= kPadEnd;
    a ^= v;
  }
  kf.permute(a);
  return a;
}

// Even and odd sums of the 4-word groups [4j, 4j + 4) for j = t0, t0 + step, ...
// < quarter: eight 16-byte loads in flight per thread.
__device__ __forceinline__ void pair_sums(const uint4* __restrict__ q, uint64_t quarter, uint64_t t0, uint64_t step, uint32_t& z, uint32_t& o) {
  for (uint64_t j = t0; j < quarter; j += 8 * step) {
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint64_t jj = j + k * step;
      v[k] = jj < quarter ? __ldg(q + jj) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      z = m31_add(z, m31_add(v[k].x, v[k].z));
      o = m31_add(o, m31_add(v[k].y, v[k].w));
    }
  }
}

// The threads that prove one table.  CtaGroup: a whole CTA (the single-table
// kernel).  PackedGroup: warps g, g + 4, g + 8, g + 12 of a 16-warp CTA, which
// the SM places on one sub-partition, with named barrier g + 1.
struct CtaGroup {
  __device__ uint32_t tid() const { return threadIdx.x; }
  __device__ uint32_t size() const { return blockDim.x; }
  __device__ void sync() const { __syncthreads(); }
};
constexpr uint32_t kPackedTables = 4;  // tables per packed CTA, one per sub-partition
constexpr uint32_t kPackedWarps = 4;   // warps per packed table
struct PackedGroup {
  uint32_t g;
  __device__ uint32_t tid() const { return (threadIdx.x >> 7) * 32 + (threadIdx.x & 31); }
  __device__ uint32_t size() const { return 32 * kPackedWarps; }
  __device__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(32 * kPackedWarps) : "memory"); }
};

// A group's shared scratch: the digest warp's exchange arrays, per-warp partial
// sums, the broadcast challenge and the digest.
struct SumcheckShared {
  __align__(16) uint64_t col[64];
  uint32_t red[2][32];
  uint32_t ch;
  uint64_t digest[4];
};

// Sum of v over the group, valid in the group's thread 0 (values < 2^31, reduced
// at every step).  Two arrays alternate, so one barrier per call suffices: thread
// 0 reads a call's array before it reaches the next call's barrier, which every
// writer of the call after that must pass first.
template <class G>
__device__ __forceinline__ uint32_t group_sum_m31(const G& grp, uint32_t v, uint32_t (&red)[2][32], uint32_t& parity) {
  for (int o = 16; o > 0; o >>= 1) v = m31_add(v, __shfl_down_sync(0xffffffffu, v, o));
  const uint32_t t = grp.tid();
  uint32_t* r = red[parity];
  parity ^= 1u;
  if ((t & 31) == 0) r[t >> 5] = v;
  grp.sync();
  uint32_t w = 0;
  if (t == 0)
    for (uint32_t k = 0; k < (grp.size() >> 5); k++) w = m31_add(w, r[k]);
  return w;
}

// One table on one group.  The group's first warp computes the statement's word
// digest while its other warps sum the table's even and odd entries (round 0's
// two sums; together the claimed sum), which need no challenge.  Then each round
// is a transcript round by the group's first warp (round frame, challenge frame,
// squeeze one word mod p) and one pass over the table that folds it,
// t'[i] = (1 - r) t[2i] + r t[2i+1], and sums the folded table's even and odd
// entries for the next round, so after the digest the table is read once per
// round.  One launch per table (or per batch of tables) leaves no launch in the
// stream waiting behind the digest, so a stream that shares a hardware work queue
// with others never holds that queue for the digest's duration.
template <class G>
__device__ void sumcheck_prove_group(const G& grp, SumcheckShared& sh, const uint32_t* __restrict__ evals, uint32_t log_n,
                                     uint32_t* __restrict__ scratch, SumcheckOut* __restrict__ out) {
  const uint64_t n = 1ull << log_n;
  const uint32_t t = grp.tid(), nt = grp.size();
  uint32_t parity = 0;
  uint32_t z = 0, o = 0;
  if (t < 32) {
    const uint64_t d = digest_words_warp(evals, n, sh.col);
    if (t < 4) sh.digest[t] = d;
  } else if (n >= 4) {
    pair_sums(reinterpret_cast<const uint4*>(evals), n >> 2, t - 32, nt - 32, z, o);
  } else if (n == 2 && t == 32) {
    z = evals[0];
    o = evals[1];
  }
  uint32_t zs = group_sum_m31(grp, z, sh.red, parity);
  uint32_t os = group_sum_m31(grp, o, sh.red, parity);
  // group_sum_m31's value is valid in thread 0, whose warp runs the transcript (the
  // digest lanes are visible to it after the first sum's barrier)
  const uint32_t total = m31_add(zs, os);
  WarpSponge sp(sh.col);
  if (t < 32) {
    if (t == 0) {
      out->claimed_sum = total;
      for (int i = 0; i < 4; i++) out->digest[i] = sh.digest[i];
    }
    uint32_t p[12] = {(uint32_t)n, (uint32_t)(n >> 32), log_n, __shfl_sync(0xffffffffu, total, 0)};
#pragma unroll
    for (int i = 0; i < 4; i++) p[4 + 2 * i] = (uint32_t)sh.digest[i], p[5 + 2 * i] = (uint32_t)(sh.digest[i] >> 32);
    sp.absorb(frame_word<SumcheckFrame>(sp.lane, 0, p));
  }
  const uint32_t* cur = evals;
  uint32_t* bufs[2] = {scratch, scratch + (n >> 1)};
  // the result arrays' addresses, read once (`out` may be host memory mapped
  // into the device's address space)
  uint32_t *r0 = nullptr, *r1 = nullptr, *chs = nullptr;
  if (t == 0) {
    r0 = out->r0;
    r1 = out->r1;
    chs = out->challenges;
  }
  for (uint32_t r = 0; r < log_n; r++) {
    const uint64_t half = (n >> r) >> 1;
    if (t < 32) {
      const uint32_t z0 = __shfl_sync(0xffffffffu, zs, 0), o0 = __shfl_sync(0xffffffffu, os, 0);
      const uint32_t pr[3] = {r, z0, o0}, pc[2] = {r, kP};
      const uint64_t fr = frame_word<SumcheckFrame>(sp.lane, 1, pr), fc = frame_word<SumcheckFrame>(sp.lane, 2, pc);
#pragma unroll 1
      for (uint32_t step = 0; step < 2; step++) sp.absorb(step == 0 ? fr : fc);
      const uint32_t c = sp.squeeze1_m31();
      if (t == 0) {
        r0[r] = z0;
        r1[r] = o0;
        chs[r] = c;
        sh.ch = c;
      }
    }
    grp.sync();
    const uint32_t c = sh.ch;
    const uint32_t omc = m31_sub(1, c);
    uint32_t* nxt = bufs[r & 1];
    z = 0;
    o = 0;
    if (half >= 2) {
      // groups of 4 entries fold into 2: 16-byte loads, 8-byte stores, 8 in flight
      const uint4* q = reinterpret_cast<const uint4*>(cur);
      uint2* w = reinterpret_cast<uint2*>(nxt);
      const uint64_t quarter = half >> 1;
      for (uint64_t j = t; j < quarter; j += 8 * (uint64_t)nt) {
        uint4 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint64_t jj = j + (uint64_t)k * nt;
          v[k] = jj < quarter ? q[jj] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint64_t jj = j + (uint64_t)k * nt;
          const uint32_t e = m31_add(m31_mul(omc, v[k].x), m31_mul(c, v[k].y));
          const uint32_t d = m31_add(m31_mul(omc, v[k].z), m31_mul(c, v[k].w));
          if (jj < quarter) {
            w[jj] = make_uint2(e, d);
            z = m31_add(z, e);
            o = m31_add(o, d);
          }
        }
      }
    } else if (t == 0) {
      nxt[0] = m31_add(m31_mul(omc, cur[0]), m31_mul(c, cur[1]));
    }
    // the sums' barriers also complete nxt (and order this round's reads of sh.ch
    // before the next round's write)
    zs = group_sum_m31(grp, z, sh.red, parity);
    os = group_sum_m31(grp, o, sh.red, parity);
    cur = nxt;
  }
  if (t == 0) out->final_eval = cur[0];
}

constexpr int kSumcheckThreads = 256;
constexpr int kPackedThreads = 32 * kPackedTables * kPackedWarps;

__global__ void __launch_bounds__(kSumcheckThreads) sumcheck_kernel(const uint32_t* __restrict__ evals, uint32_t log_n, uint32_t* __restrict__ scratch,
                                                                  SumcheckOut* __restrict__ out) {
  __shared__ SumcheckShared sh;
  sumcheck_prove_group(CtaGroup{}, sh, evals, log_n, scratch, out);
}

// Up to four tables per CTA, table g on warps g, g + 4, g + 8, g + 12: the SM
// places a CTA's warps on its four sub-partitions in turn, so the four digest
// warps get a sub-partition each, beside only their own table's three summing
// warps (which wait at the first barrier once round 0's sums are done), never
// beside another of the CTA's digests.
__global__ void __launch_bounds__(kPackedThreads, 1) sumcheck_packed_kernel(const __grid_constant__ SumcheckBatch batch, uint32_t count) {
  __shared__ SumcheckShared sh[kPackedTables];
  const uint32_t g = (threadIdx.x >> 5) & (kPackedTables - 1);
  const uint32_t k = blockIdx.x * kPackedTables + g;
  if (k >= count) return;  // the group's warps all leave; no other group waits on them
  const SumcheckJob& j = batch.job[k];
  sumcheck_prove_group(PackedGroup{g}, sh[g], j.evals, j.log_n, j.scratch, j.out);
}

cudaError_t launch_sumcheck(const uint32_t* evals, uint32_t log_n, uint32_t* scratch, SumcheckOut* out, cudaStream_t s) {
  sumcheck_kernel<<<1, kSumcheckThreads, 0, s>>>(evals, log_n, scratch, out);
  return cudaGetLastError();
}

cudaError_t launch_sumcheck_batch(const SumcheckBatch& batch, uint32_t count, cudaStream_t s) {
  if (!count) return cudaSuccess;
  if (count > kSumcheckBatchMax) return cudaErrorInvalidValue;
  sumcheck_packed_kernel<<<(count + kPackedTables - 1) / kPackedTables, kPackedThreads, 0, s>>>(batch, count);
  return cudaGetLastError();
}

}  // namespace azk

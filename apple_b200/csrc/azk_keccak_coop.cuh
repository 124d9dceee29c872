// Keccak-f[1600] spread over several lanes, for work that has too few
// permutations to hide one thread's latency: the upper levels of a Merkle tree,
// small trees, the transcript and the sum-check's sequential digest.
//
// Measured on B200 (one SM at 1.965 GHz, chains of dependent permutations, cycles
// per round at 1 / 2 / 4 warps per SM sub-partition):
//   one thread each       370 / 720 / 1441   (32 permutations per warp)
//   a pair of lanes each  226 / 372 /  734   (16 permutations per warp)
//   a warp each           186 / 238 /  466   (1 permutation per warp)
// A permutation by one thread is bound by the issue of its 180 logic and shift
// instructions per round (two cycles each on the half-rate integer pipe); a pair
// halves them and pays 17 shuffles, which run on another pipe, so its throughput
// stays within 2-7 % of the one-thread form while its latency drops to 0.61; a
// whole warp is bound by the latency of its two exchanges per round.
#pragma once
#include <stdint.h>

#include "azk_keccak.cuh"

namespace azk {

// ---------------------------------------------------------------------------
// Bit interleaving: a 64-bit lane as the word of its even bits and the word of its
// odd bits.  A rotation of the lane by r then is a rotation of each word by r / 2
// (r even), or the two words exchanged and rotated by (r + 1) / 2 (the new even
// word) and (r - 1) / 2 (the new odd word).
// ---------------------------------------------------------------------------
// Even bits of each 16-bit half of x to its low byte, odd bits to its high byte (and
// back), by exchanging neighbouring fields of doubling width (the unshuffle of H. S.
// Warren, Hacker's Delight, 7-2); the bytes of both words of a lane then move in two
// permutes.
__host__ __device__ __forceinline__ uint32_t unshuffle16(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 1)) & 0x22222222u; x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu; x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u; x ^= t ^ (t << 4);
  return x;
}
__host__ __device__ __forceinline__ uint32_t shuffle16(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 4)) & 0x00F000F0u; x ^= t ^ (t << 4);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu; x ^= t ^ (t << 2);
  t = (x ^ (x >> 1)) & 0x22222222u; x ^= t ^ (t << 1);
  return x;
}
// Bytes 0..3 are a's, 4..7 are b's; digit k of `sel` picks the result's byte k.
template <uint32_t SEL>
__host__ __device__ __forceinline__ uint32_t pick_bytes(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(a, b, SEL);
#else
  const uint64_t v = ((uint64_t)b << 32) | a;
  uint32_t r = 0;
  for (int k = 0; k < 4; k++) r |= (uint32_t)((v >> (8 * ((SEL >> (4 * k)) & 7))) & 0xFF) << (8 * k);
  return r;
#endif
}
__host__ __device__ __forceinline__ void split64(uint64_t v, uint32_t& even, uint32_t& odd) {
  const uint32_t lo = unshuffle16((uint32_t)v), hi = unshuffle16((uint32_t)(v >> 32));
  even = pick_bytes<0x6420>(lo, hi);
  odd = pick_bytes<0x7531>(lo, hi);
}
__host__ __device__ __forceinline__ uint64_t join64(uint32_t even, uint32_t odd) {
  const uint32_t lo = shuffle16(pick_bytes<0x5140>(even, odd)), hi = shuffle16(pick_bytes<0x7362>(even, odd));
  return ((uint64_t)hi << 32) | lo;
}

// Round constants in split form.
struct alignas(8) SplitRC {
  uint32_t even, odd;
};
struct KeccakSplitRC {
  SplitRC w[24];
};
constexpr uint32_t keccak_every_second_bit(uint64_t v) {
  uint32_t r = 0;
  for (int i = 0; i < 32; i++) r |= (uint32_t)((v >> (2 * i)) & 1) << i;
  return r;
}
constexpr KeccakSplitRC keccak_split_rc() {
  const uint64_t rc[24] = {0x0000000000000001ULL, 0x0000000000008082ULL, 0x800000000000808AULL, 0x8000000080008000ULL, 0x000000000000808BULL,
                           0x0000000080000001ULL, 0x8000000080008081ULL, 0x8000000000008009ULL, 0x000000000000008AULL, 0x0000000000000088ULL,
                           0x0000000080008009ULL, 0x000000008000000AULL, 0x000000008000808BULL, 0x800000000000008BULL, 0x8000000000008089ULL,
                           0x8000000000008003ULL, 0x8000000000008002ULL, 0x8000000000000080ULL, 0x000000000000800AULL, 0x800000008000000AULL,
                           0x8000000080008081ULL, 0x8000000000008080ULL, 0x0000000080000001ULL, 0x8000000080008008ULL};
  KeccakSplitRC r{};
  for (int i = 0; i < 24; i++) r.w[i] = SplitRC{keccak_every_second_bit(rc[i]), keccak_every_second_bit(rc[i] >> 1)};
  return r;
}
__constant__ static const KeccakSplitRC kKeccakSplitRC = keccak_split_rc();

// ---------------------------------------------------------------------------
// One thread per permutation, in split form: theta's rotation by one moves a word
// (5 shifts a round instead of 10) and so does lane 1's, so a round is 174
// instructions instead of 180.  For 16-byte messages and digests that stay in split
// form; splitting and joining a digest costs 104.
// ---------------------------------------------------------------------------
struct SplitDigest {
  uint4 even, odd;  // four lanes
};
template <int R>
__device__ __forceinline__ void split_rotl(uint32_t e, uint32_t o, uint32_t& re, uint32_t& ro) {
  if constexpr (R & 1) {
    re = __funnelshift_l(o, o, (R + 1) / 2);
    ro = __funnelshift_l(e, e, R / 2);
  } else {
    re = __funnelshift_l(e, e, R / 2);
    ro = __funnelshift_l(o, o, R / 2);
  }
}
// D of column x is c[x - 1] ^ rotl(c[x + 1], 1): r[x] holds the rotated even words
// (the rotated odd words are ce).  Lanes outside NZ are zero.
template <uint32_t NZ, int I>
__device__ __forceinline__ void split_rho_pi_lane(const uint32_t (&e)[25], const uint32_t (&o)[25], const uint32_t (&ce)[5], const uint32_t (&co)[5],
                                                  const uint32_t (&r)[5], uint32_t (&be)[25], uint32_t (&bo)[25]) {
  constexpr int m = (I % 5 + 4) % 5, n = (I % 5 + 1) % 5;
  uint32_t te, to;
  if constexpr ((NZ >> I) & 1u) {
    te = lop3_xor3(e[I], ce[m], r[n]);
    to = lop3_xor3(o[I], co[m], ce[n]);
  } else {
    te = ce[m] ^ r[n];
    to = co[m] ^ ce[n];
  }
  split_rotl<RhoPi<I>::rho>(te, to, be[RhoPi<I>::dst], bo[RhoPi<I>::dst]);
}
template <uint32_t NZ, int... Is>
__device__ __forceinline__ void split_rho_pi(const uint32_t (&e)[25], const uint32_t (&o)[25], const uint32_t (&ce)[5], const uint32_t (&co)[5],
                                             const uint32_t (&r)[5], uint32_t (&be)[25], uint32_t (&bo)[25], LaneSeq<Is...>) {
  (split_rho_pi_lane<NZ, Is>(e, o, ce, co, r, be, bo), ...);
}
template <uint32_t NZ>
__device__ __forceinline__ void split_columns(const uint32_t (&a)[25], uint32_t (&c)[5]) {
#pragma unroll
  for (int x = 0; x < 5; x++) {
    if constexpr (NZ == kLanesAll) {
      c[x] = lop3_xor3(lop3_xor3(a[x], a[x + 5], a[x + 10]), a[x + 15], a[x + 20]);
    } else {
      c[x] = 0;
#pragma unroll
      for (int i = x; i < 25; i += 5)
        if ((NZ >> i) & 1u) c[x] ^= a[i];
    }
  }
}
template <uint32_t NZ>
__device__ __forceinline__ void split_round(uint32_t (&e)[25], uint32_t (&o)[25], int round) {
  uint32_t ce[5], co[5], r[5], be[25], bo[25];
  split_columns<NZ>(e, ce);
  split_columns<NZ>(o, co);
#pragma unroll
  for (int x = 0; x < 5; x++) r[x] = __funnelshift_l(co[x], co[x], 1);
  split_rho_pi<NZ>(e, o, ce, co, r, be, bo, LaneSeq<0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24>{});
#pragma unroll
  for (int y = 0; y < 25; y += 5) {
#pragma unroll
    for (int x = 0; x < 5; x++) {
      e[y + x] = lop3_chi(be[y + x], be[y + (x + 1) % 5], be[y + (x + 2) % 5]);
      o[y + x] = lop3_chi(bo[y + x], bo[y + (x + 1) % 5], bo[y + (x + 2) % 5]);
    }
  }
  e[0] ^= kKeccakSplitRC.w[round].even;
  o[0] ^= kKeccakSplitRC.w[round].odd;
}
// Rounds 1 .. 23 of a one-block digest (see keccak_digest).
__device__ __forceinline__ SplitDigest split_digest_rest(uint32_t (&e)[25], uint32_t (&o)[25]) {
#pragma unroll 1
  for (int i = 1; i < 23; i += 2) {
    split_round<kLanesAll>(e, o, i);
    split_round<kLanesAll>(e, o, i + 1);
  }
  uint32_t ce[5], co[5], r[5], be[25], bo[25];
  split_columns<kLanesAll>(e, ce);
  split_columns<kLanesAll>(o, co);
#pragma unroll
  for (int x = 0; x < 5; x++) r[x] = __funnelshift_l(co[x], co[x], 1);
  split_rho_pi<kLanesAll>(e, o, ce, co, r, be, bo, LaneSeq<0, 6, 12, 18, 24>{});
  return {make_uint4(lop3_chi(be[0], be[1], be[2]) ^ kKeccakSplitRC.w[23].even, lop3_chi(be[1], be[2], be[3]), lop3_chi(be[2], be[3], be[4]),
                     lop3_chi(be[3], be[4], be[0])),
          make_uint4(lop3_chi(bo[0], bo[1], bo[2]) ^ kKeccakSplitRC.w[23].odd, lop3_chi(bo[1], bo[2], bo[3]), lop3_chi(bo[2], bo[3], bo[4]),
                     lop3_chi(bo[3], bo[4], bo[0]))};
}

// ---------------------------------------------------------------------------
// A pair of neighbouring lanes per permutation.  Lane parity q = 0 holds the 25
// even words, q = 1 the 25 odd words.  Every lane of the warp takes part (the
// exchanges are full-warp shuffles), so callers keep warps converged and clamp the
// indices of lanes without work.
// ---------------------------------------------------------------------------
// One uniform 8-byte load and a select: loads indexed or predicated by the lane's
// parity cost a round 10 cycles.
__device__ __forceinline__ uint32_t split_rc(int r, uint32_t q) {
  const uint2 v = reinterpret_cast<const uint2*>(kKeccakSplitRC.w)[r];
  return q ? v.y : v.x;
}

template <int I>
__device__ __forceinline__ void pair_rho_pi_lane(const uint32_t (&a)[25], const uint32_t (&c)[5], const uint32_t (&r1)[5], uint32_t (&b)[25], uint32_t q) {
  constexpr int x = I % 5, r = RhoPi<I>::rho;
  uint32_t t = lop3_xor3(a[I], c[(x + 4) % 5], r1[(x + 1) % 5]);
  if constexpr (r & 1) {
    t = __shfl_xor_sync(0xffffffffu, t, 1);
    t = __funnelshift_l(t, t, (uint32_t)((r + 1) / 2) - q);
  } else if constexpr (r != 0) {
    t = __funnelshift_l(t, t, r / 2);
  }
  b[RhoPi<I>::dst] = t;
}
template <int... Is>
__device__ __forceinline__ void pair_rho_pi(const uint32_t (&a)[25], const uint32_t (&c)[5], const uint32_t (&r1)[5], uint32_t (&b)[25], uint32_t q,
                                            LaneSeq<Is...>) {
  (pair_rho_pi_lane<Is>(a, c, r1, b, q), ...);
}
__device__ __forceinline__ void pair_round(uint32_t (&a)[25], uint32_t q, uint32_t rc) {
  uint32_t c[5], r1[5], b[25];
#pragma unroll
  for (int x = 0; x < 5; x++) c[x] = lop3_xor3(lop3_xor3(a[x], a[x + 5], a[x + 10]), a[x + 15], a[x + 20]);
#pragma unroll
  for (int x = 0; x < 5; x++) {
    const uint32_t p = __shfl_xor_sync(0xffffffffu, c[x], 1);
    r1[x] = __funnelshift_l(p, p, 1u - q);
  }
  // the odd rotations (which exchange words) first, the even ones under their latency
  pair_rho_pi(a, c, r1, b, q, LaneSeq<1, 4, 8, 10, 12, 13, 14, 15, 16, 17, 18, 22, 0, 2, 3, 5, 6, 7, 9, 11, 19, 20, 21, 23, 24>{});
#pragma unroll
  for (int y = 0; y < 25; y += 5) {
#pragma unroll
    for (int x = 0; x < 5; x++) a[y + x] = lop3_chi(b[y + x], b[y + (x + 1) % 5], b[y + (x + 2) % 5]);
  }
  a[0] ^= rc;
}
// Two rounds per iteration: one costs 6 % more latency at a warp per sub-partition.
__device__ __forceinline__ void pair_f1600(uint32_t (&a)[25], uint32_t q) {
#pragma unroll 1
  for (int r = 0; r < 24; r += 2) {
    pair_round(a, q, split_rc(r, q));
    pair_round(a, q, split_rc(r + 1, q));
  }
}

// The one-block digest of azk_keccak.cuh (keccak_digest) by a pair: the first round
// without the zero lanes, the last without what its row 0 does not need.
template <uint32_t NZ, int I>
__device__ __forceinline__ void pair_rho_pi_first_lane(const uint32_t (&a)[25], const uint32_t (&c)[5], const uint32_t (&r1)[5], const uint32_t (&d)[5],
                                                       uint32_t (&b)[25], uint32_t q) {
  constexpr int x = I % 5, r = RhoPi<I>::rho;
  uint32_t t;
  if constexpr ((NZ >> I) & 1u) t = lop3_xor3(a[I], c[(x + 4) % 5], r1[(x + 1) % 5]);
  else t = d[x];
  if constexpr (r & 1) {
    t = __shfl_xor_sync(0xffffffffu, t, 1);
    t = __funnelshift_l(t, t, (uint32_t)((r + 1) / 2) - q);
  } else if constexpr (r != 0) {
    t = __funnelshift_l(t, t, r / 2);
  }
  b[RhoPi<I>::dst] = t;
}
template <uint32_t NZ, int... Is>
__device__ __forceinline__ void pair_rho_pi_first(const uint32_t (&a)[25], const uint32_t (&c)[5], const uint32_t (&r1)[5], const uint32_t (&d)[5],
                                                  uint32_t (&b)[25], uint32_t q, LaneSeq<Is...>) {
  (pair_rho_pi_first_lane<NZ, Is>(a, c, r1, d, b, q), ...);
}
template <uint32_t NZ>
__device__ __forceinline__ uint4 pair_digest(uint32_t (&a)[25], uint32_t q) {
  uint32_t c[5], r1[5], d[5], b[25];
#pragma unroll
  for (int x = 0; x < 5; x++) {
    c[x] = 0;
#pragma unroll
    for (int i = x; i < 25; i += 5)
      if ((NZ >> i) & 1u) c[x] ^= a[i];
  }
#pragma unroll
  for (int x = 0; x < 5; x++) {
    const uint32_t p = __shfl_xor_sync(0xffffffffu, c[x], 1);
    r1[x] = __funnelshift_l(p, p, 1u - q);
  }
#pragma unroll
  for (int x = 0; x < 5; x++) d[x] = c[(x + 4) % 5] ^ r1[(x + 1) % 5];
  pair_rho_pi_first<NZ>(a, c, r1, d, b, q, LaneSeq<1, 4, 8, 10, 12, 13, 14, 15, 16, 17, 18, 22, 0, 2, 3, 5, 6, 7, 9, 11, 19, 20, 21, 23, 24>{});
#pragma unroll
  for (int y = 0; y < 25; y += 5) {
#pragma unroll
    for (int x = 0; x < 5; x++) a[y + x] = lop3_chi(b[y + x], b[y + (x + 1) % 5], b[y + (x + 2) % 5]);
  }
  a[0] ^= split_rc(0, q);
#pragma unroll 1
  for (int r = 1; r < 23; r += 2) {
    pair_round(a, q, split_rc(r, q));
    pair_round(a, q, split_rc(r + 1, q));
  }
#pragma unroll
  for (int x = 0; x < 5; x++) c[x] = lop3_xor3(lop3_xor3(a[x], a[x + 5], a[x + 10]), a[x + 15], a[x + 20]);
#pragma unroll
  for (int x = 0; x < 5; x++) {
    const uint32_t p = __shfl_xor_sync(0xffffffffu, c[x], 1);
    r1[x] = __funnelshift_l(p, p, 1u - q);
  }
  pair_rho_pi(a, c, r1, b, q, LaneSeq<12, 18, 0, 6, 24>{});
  return make_uint4(lop3_chi(b[0], b[1], b[2]) ^ split_rc(23, q), lop3_chi(b[1], b[2], b[3]), lop3_chi(b[2], b[3], b[4]), lop3_chi(b[3], b[4], b[0]));
}

// Split form of small padding constants: suffix 0x06 or 0x01 in the lowest byte of
// a lane, 0x80 in its highest byte.
__device__ __forceinline__ uint32_t pair_suffix(uint32_t suffix, uint32_t q) {
  return suffix == 0x06 ? (q ? 1u : 2u) : (q ? 0u : 1u);
}
__device__ __forceinline__ uint32_t pair_pad_end(uint32_t q) { return q ? 0x80000000u : 0u; }

// Lane i owned by the pair's thread 0 and lane j owned by its thread 1 (`mine` is
// the caller's): each thread gets its own parity's words of both.
__device__ __forceinline__ void pair_split2(uint64_t mine, uint32_t q, uint32_t& wi, uint32_t& wj) {
  uint32_t e, o;
  split64(mine, e, o);
  const uint32_t got = __shfl_xor_sync(0xffffffffu, q ? e : o, 1);
  wi = q ? got : e;
  wj = q ? o : got;
}
// A 32-byte digest in memory (four lanes) as this thread's parity's four words.
__device__ __forceinline__ uint4 pair_split_digest(ulonglong2 half, uint32_t q) {  // half: lanes 2q, 2q + 1
  uint4 v;
  pair_split2(half.x, q, v.x, v.z);
  pair_split2(half.y, q, v.y, v.w);
  return v;
}
// The reverse: lanes 2q and 2q + 1 of the digest whose split words the pair holds.
__device__ __forceinline__ ulonglong2 pair_join_digest(uint4 v, uint32_t q) {
  const uint32_t g0 = __shfl_xor_sync(0xffffffffu, q ? v.x : v.z, 1), g1 = __shfl_xor_sync(0xffffffffu, q ? v.y : v.w, 1);
  return q ? make_ulonglong2(join64(g0, v.z), join64(g1, v.w)) : make_ulonglong2(join64(v.x, g0), join64(v.y, g1));
}
// SHA3-256 of two digests (a Merkle parent), all in split form.
__device__ __forceinline__ uint4 pair_hash_parent(uint4 l, uint4 r, uint32_t q) {
  uint32_t a[25];
  a[0] = l.x, a[1] = l.y, a[2] = l.z, a[3] = l.w;
  a[4] = r.x, a[5] = r.y, a[6] = r.z, a[7] = r.w;
  a[8] = pair_suffix(0x06, q);
  a[16] = pair_pad_end(q);
  return pair_digest<kLanes64>(a, q);
}

// ---------------------------------------------------------------------------
// One warp per permutation: what counts is the latency of a chain of dependent
// permutations.  Lane x + 5y (< 25) holds state lane (x, y); lanes 25..31 follow
// lane 0's indices and store nothing.  A round is two exchanges, and its cost
// follows the number of exchange instructions more than the number of dependent
// stages (measured on B200: three shuffle stages 2.43 us per permutation, two
// shuffle stages 2.30 us, this form 1.98 us):
//   1. every lane stores its lane into a column-major shared array (columns
//      padded to 6 words so a column is two 16-byte loads and one 8-byte load)
//      and reads columns x - 1 and x + 1: theta's D[x], then rho's rotation of
//      its own lane, e = rotl(a ^ D[x], rho[x, y]), at the source.  Rounds
//      alternate between two arrays, so the one __syncwarp after the stores also
//      orders the previous round's loads of the other array before its next stores;
//   2. pi and chi in one gather: lane (x, y) shuffles e from the pi sources of
//      (x, y), (x + 1, y) and (x + 2, y); iota enters as chi(b0 ^ rc, b1, b2)
//      (= chi(b0, b1, b2) ^ rc) through a mask that is zero except on lane 0, so
//      its XOR overlaps the wait for the later shuffles.
// ---------------------------------------------------------------------------
__constant__ static const uint8_t kRhoOffsets[25] = {0,  1,  62, 28, 27, 36, 44, 6,  55, 20, 3,  10, 43,
                                                     25, 39, 41, 45, 15, 21, 8,  18, 2,  61, 56, 14};

struct WarpKeccak {
  uint64_t* col;        // two arrays of 5 columns x 6 words, column-major (16-byte aligned)
  uint32_t own;         // this lane's word in col
  uint32_t cm, cp;      // first words of columns x - 1 and x + 1
  uint32_t s0, s1, s2;  // pi sources of (x, y), (x + 1, y), (x + 2, y)
  uint32_t swap, rot;   // rho[x, y] as a half swap (bit 5) and a funnel shift
  uint64_t rc_mask;     // all ones on lane 0
  bool stores;

  __device__ __forceinline__ WarpKeccak(uint32_t lane, uint64_t* smem) : col(smem) {
    const uint32_t t = lane < 25 ? lane : 0;
    const uint32_t x = t % 5, y = t / 5;
    own = 6 * x + y;
    cm = 6 * ((x + 4) % 5);
    cp = 6 * ((x + 1) % 5);
    // B[X, Y] = rotl(A'[xs, ys]) with X = ys, Y = 2 xs + 3 ys (mod 5); 2^-1 = 3 (mod 5)
    auto src = [](uint32_t X, uint32_t Y) { return (((Y + 15 - 3 * X) % 5) * 3) % 5 + 5 * X; };
    s0 = src(x, y);
    s1 = src((x + 1) % 5, y);
    s2 = src((x + 2) % 5, y);
    const uint32_t r = kRhoOffsets[t];
    swap = r & 32u;
    rot = r & 31u;
    rc_mask = lane == 0 ? ~0ull : 0ull;
    stores = lane < 25;
  }

  __device__ __forceinline__ void round(uint64_t& a, uint64_t* c, uint64_t rc) const {
    if (stores) c[own] = a;
    __syncwarp();
    const ulonglong2 m01 = *reinterpret_cast<const ulonglong2*>(c + cm);
    const ulonglong2 m23 = *reinterpret_cast<const ulonglong2*>(c + cm + 2);
    const uint64_t m4 = c[cm + 4];
    const ulonglong2 p01 = *reinterpret_cast<const ulonglong2*>(c + cp);
    const ulonglong2 p23 = *reinterpret_cast<const ulonglong2*>(c + cp + 2);
    const uint64_t p4 = c[cp + 4];
    const uint64_t c_m = xor3_64(xor3_64(m01.x, m01.y, m23.x), m23.y, m4);
    const uint64_t c_p = xor3_64(xor3_64(p01.x, p01.y, p23.x), p23.y, p4);
    const uint64_t t = xor3_64(a, c_m, rotl<1>(c_p));
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32);
    const uint32_t l2 = swap ? hi : lo, h2 = swap ? lo : hi;
    const uint64_t e = ((uint64_t)__funnelshift_l(l2, h2, rot) << 32) | __funnelshift_l(h2, l2, rot);
    const uint64_t b0 = __shfl_sync(0xffffffffu, e, s0) ^ (rc & rc_mask);
    const uint64_t b1 = __shfl_sync(0xffffffffu, e, s1);
    const uint64_t b2 = __shfl_sync(0xffffffffu, e, s2);
    a = chi_64(b0, b1, b2);
  }

  // All 24 rounds unrolled: the round constants are immediates (the sum-check's
  // chain of thousands of permutations).
  __device__ __forceinline__ void permute(uint64_t& a) const {
#pragma unroll
    for (int r = 0; r < 24; r += 8) {
#pragma unroll
      for (int k = 0; k < 8; k++) round(a, col + 32 * (k & 1), kKeccakRC[r + k]);
    }
  }
  // Four rounds per iteration: for kernels that permute a few times in several places.
  __device__ __forceinline__ void permute_small(uint64_t& a) const {
#pragma unroll 1
    for (int r = 0; r < 24; r += 4) {
#pragma unroll
      for (int k = 0; k < 4; k++) round(a, col + 32 * (k & 1), kKeccakRC[r + k]);
    }
  }
};

static constexpr uint32_t kWarpKeccakWords = 64;  // u64 words of shared exchange space per warp

}  // namespace azk

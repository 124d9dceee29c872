// Loading fixed-rate messages (<= 136 bytes) into a Keccak state and hashing them
// with SHA3-256 (suffix 0x06) or Keccak-256 (suffix 0x01), as the reference's
// one-block kernels do (HashMerkleKernels.metal:584-909): a message shorter than
// the rate is one permutation; a 136-byte message fills the first block and the
// padding takes a second permutation (absorb_fixed_136, :633-657).
#pragma once
#include "azk_keccak.cuh"

namespace azk {

// 64-bit words of a message at any byte address, from aligned 4-byte loads and
// funnel shifts.  Only 4-byte units that hold message bytes are read (they lie inside
// the message's allocation).  Byte loads were four times as many requests (2^20
// messages of 99 bytes at stride 102, 256 threads per CTA: 354 us with byte loads,
// 287 us so; 64 threads: 277 and 267).
struct UnalignedWords {
  const uint32_t* q;
  uint32_t off;  // bytes from *q to the message
  __device__ __forceinline__ explicit UnalignedWords(const uint8_t* p)
      : q(reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3)), off((uint32_t)reinterpret_cast<uintptr_t>(p) & 3u) {}
  // Bytes 8i .. 8i + n - 1 of the message (1 <= n <= 8), zeros above them.
  __device__ __forceinline__ uint64_t word(uint32_t i, uint32_t n) const {
    const uint32_t* w = q + 2 * i;
    const uint32_t end = off + n, sh = 8 * off;
    const uint32_t w0 = __ldg(w), w1 = end > 4 ? __ldg(w + 1) : 0u, w2 = end > 8 ? __ldg(w + 2) : 0u;
    const uint64_t v = ((uint64_t)__funnelshift_r(w1, w2, sh) << 32) | __funnelshift_r(w0, w1, sh);
    return n == 8 ? v : v & ((1ull << (8 * n)) - 1);
  }
};

// XOR `len` message bytes into lanes 0..16.  aligned8: p is 8-byte aligned, so
// whole lanes load as u64.
__device__ __forceinline__ void xor_message(uint64_t (&a)[25], const uint8_t* p, uint32_t len, bool aligned8) {
  const uint32_t full = len >> 3, rem = len & 7;
  const UnalignedWords u(p);
  if (aligned8) {
    const uint64_t* q = reinterpret_cast<const uint64_t*>(p);
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i < full) a[i] ^= __ldg(q + i);
  } else {
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i < full) a[i] ^= u.word(i, 8);
  }
  if (rem) {
    const uint64_t v = u.word(full, rem);
    // lane index `full` is dynamic here; select it with an unrolled compare
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i == full) a[i] ^= v;
  }
}

// Digest of one message of `len` (<= 136) bytes at p.
__device__ __forceinline__ void hash_message(const uint8_t* p, uint32_t len, uint32_t suffix, bool aligned8, uint64_t (&out)[4]) {
  uint64_t a[25];
#pragma unroll
  for (int i = 0; i < 25; i++) a[i] = 0;
  xor_message(a, p, len, aligned8);
  if (len == 136) {
    keccak_f1600(a);
    a[0] ^= suffix;
    a[16] ^= kPadEnd;
    keccak_digest<kLanesAll>(a, out);
  } else {
    uint32_t lane = len >> 3;
    uint64_t v = (uint64_t)suffix << (8 * (len & 7));
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i == lane) a[i] ^= v;
    a[16] ^= kPadEnd;
    keccak_digest<kLanesRate>(a, out);
  }
}

}  // namespace azk

// Loading fixed-rate messages (<= 136 bytes) into a Keccak state and hashing them
// with SHA3-256 (suffix 0x06) or Keccak-256 (suffix 0x01), as the reference's
// one-block kernels do (HashMerkleKernels.metal:584-909): a message shorter than
// the rate is one permutation; a 136-byte message fills the first block and the
// padding takes a second permutation (absorb_fixed_136, :633-657).
#pragma once
#include <string.h>

#include "azk_keccak.cuh"

namespace azk {

// Loads of read-only message memory (a parameter of the readers below, so that the
// addresses they touch can be checked on the host).
struct ReadOnlyLoads {
  template <class T>
  __host__ __device__ __forceinline__ static T load(const uint8_t* p) {
#if defined(__CUDA_ARCH__)
    return __ldg(reinterpret_cast<const T*>(p));
#else
    T v;
    memcpy(&v, p, sizeof(T));
    return v;
#endif
  }
};

// Loads of a message in global or shared memory.
struct AnyLoads {
  template <class T>
  __host__ __device__ __forceinline__ static T load(const uint8_t* p) {
    return *reinterpret_cast<const T*>(p);
  }
};

// Bytes [from, to) of the 4-byte unit at q (4-byte aligned), in their places, zeros
// around them; no other byte is read.
template <class L>
__host__ __device__ __forceinline__ uint32_t unit_bytes(const uint8_t* q, uint32_t from, uint32_t to) {
  uint32_t v = 0;
  if (from == 0 && to >= 2) v = L::template load<uint16_t>(q);
  else if (from == 0 && to == 1) v = L::template load<uint8_t>(q);
  else if (from == 1 && to >= 2) v = (uint32_t)L::template load<uint8_t>(q + 1) << 8;
  if (from <= 2 && to == 4) v |= (uint32_t)L::template load<uint16_t>(q + 2) << 16;
  else if (from <= 2 && to == 3) v |= (uint32_t)L::template load<uint8_t>(q + 2) << 16;
  else if (from == 3 && to == 4) v |= (uint32_t)L::template load<uint8_t>(q + 3) << 24;
  return v;
}

// The last n (1 .. 7) bytes of a message whose words are 8-byte aligned.
template <class L = ReadOnlyLoads>
__host__ __device__ __forceinline__ uint64_t aligned_tail(const uint8_t* p, uint32_t n) {
  uint64_t v = 0;
  if (n & 4) v = L::template load<uint32_t>(p);
  if (n & 2) v |= (uint64_t)L::template load<uint16_t>(p + (n & 4)) << (8 * (n & 4));
  if (n & 1) v |= (uint64_t)L::template load<uint8_t>(p + (n & 6)) << (8 * (n & 6));
  return v;
}

// 64-bit words of a message at any byte address, from aligned 4-byte loads and
// shifts.  EDGE: units that are not all message are taken by bytes and halves, so no byte
// outside the message is read (raw leaves: a select more per word).  Otherwise they are
// taken whole and masked; hash_batch keeps such units inside its buffers.
template <bool EDGE, class L = ReadOnlyLoads>
struct UnalignedWords {
  const uint8_t* q;     // the unit that holds the first byte
  uint32_t off;         // bytes from q to the message
  uint32_t last = ~0u;  // EDGE: index of a last unit that is not all message,
  uint32_t head = 0, tail = 0;  // the first unit's message bytes, and that one's
  __host__ __device__ __forceinline__ UnalignedWords(const uint8_t* p, uint32_t len) : off((uint32_t)reinterpret_cast<uintptr_t>(p) & 3u) {
    q = p - off;
    if constexpr (EDGE) {
      const uint32_t end = off + len;
      head = off == 0 && end >= 4 ? L::template load<uint32_t>(q) : unit_bytes<L>(q, off, end < 4 ? end : 4);
      if (end > 4 && (end & 3)) {
        last = end >> 2;
        tail = unit_bytes<L>(q + 4 * last, 0, end & 3);
      }
    }
  }
  __host__ __device__ __forceinline__ uint32_t unit(uint32_t k) const {
    if constexpr (EDGE)
      if (k == 0 || k == last) return k == 0 ? head : tail;
    return L::template load<uint32_t>(q + 4 * k);
  }
  // Bytes 8i .. 8i + n - 1 of the message (1 <= n <= 8), zeros above them.
  __host__ __device__ __forceinline__ uint64_t word(uint32_t i, uint32_t n) const {
    const uint32_t end = off + n;
    const uint32_t w0 = unit(2 * i), w1 = end > 4 ? unit(2 * i + 1) : 0u, w2 = end > 8 ? unit(2 * i + 2) : 0u;
#if defined(__CUDA_ARCH__)
    const uint32_t sh = 8 * off;
    const uint64_t v = ((uint64_t)__funnelshift_r(w1, w2, sh) << 32) | __funnelshift_r(w0, w1, sh);
#else
    const uint64_t lo = ((uint64_t)w1 << 32) | w0;
    const uint64_t v = off ? (lo >> (8 * off)) | ((uint64_t)w2 << (64 - 8 * off)) : lo;
#endif
    return n == 8 ? v : v & ((1ull << (8 * n)) - 1);
  }
};

// XOR `len` message bytes into lanes 0..16.  aligned8: p is 8-byte aligned, so
// whole lanes load as u64.  EDGE, L: see UnalignedWords; LA: the loads of aligned ones.
template <bool EDGE, class L = ReadOnlyLoads, class LA = L>
__host__ __device__ __forceinline__ void xor_message(uint64_t (&a)[25], const uint8_t* p, uint32_t len, bool aligned8) {
  const uint32_t full = len >> 3, rem = len & 7;
  uint64_t v = 0;
  if (aligned8) {
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i < full) a[i] ^= LA::template load<uint64_t>(p + 8 * i);
    if (rem) v = aligned_tail<LA>(p + 8 * full, rem);
  } else {
    const UnalignedWords<EDGE, L> u(p, len);
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i < full) a[i] ^= u.word(i, 8);
    if (rem) v = u.word(full, rem);
  }
  if (rem) {
    // lane index `full` is dynamic here; select it with an unrolled compare
#pragma unroll
    for (uint32_t i = 0; i < 17; i++)
      if (i == full) a[i] ^= v;
  }
}

#if defined(__CUDACC__)
// Digest of one message of `len` (<= 136) bytes at p.
template <bool EDGE, class L = ReadOnlyLoads, class LA = L>
__device__ __forceinline__ void hash_message(const uint8_t* p, uint32_t len, uint32_t suffix, bool aligned8, uint64_t (&out)[4]) {
  uint64_t a[25];
#pragma unroll
  for (int i = 0; i < 25; i++) a[i] = 0;
  xor_message<EDGE, L, LA>(a, p, len, aligned8);
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
#endif

}  // namespace azk

// SHA3 Merkle commitment kernels: fused leaf hashing + shared-memory treelets +
// last-arriver upper levels, for raw leaves, prehashed digests, QM31 layers and
// fold-then-hash layers with 16-byte leaves of one QM31 value or 64-byte leaves of
// four (reference: MerkleCommitter.swift:526-1063 and the Metal
// kernels HashMerkleKernels.metal:1064-1292; oracle MerkleOracle.swift:4-141).
//
// Tree layout: level 0 (leaf digests) optional; levels >= 1 in `inner`, level l
// at inner_offset(logn, l), root last.  A digest is 4 little-endian u64 lanes.
//
// Upper levels need no grid-wide wait: each CTA that completes a treelet root
// bumps its group's arrival counter; the CTA that arrives last reads the group's
// roots (written by the others before their fence + atomic) and reduces them.
// Counters reset themselves, so the same job list can be relaunched (and
// captured in a CUDA graph).
#include "azk_field.cuh"
#include "azk_internal.h"
#include "azk_message.cuh"
#include "azk_transcript_warp.cuh"

namespace azk {

__device__ __forceinline__ void st_dig(uint64_t* p, const uint64_t (&d)[4]) {
  reinterpret_cast<ulonglong2*>(p)[0] = make_ulonglong2(d[0], d[1]);
  reinterpret_cast<ulonglong2*>(p)[1] = make_ulonglong2(d[2], d[3]);
}
__device__ __forceinline__ void ld_dig(const uint64_t* p, uint64_t (&d)[4]) {
  ulonglong2 a = reinterpret_cast<const ulonglong2*>(p)[0], b = reinterpret_cast<const ulonglong2*>(p)[1];
  d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
}
// L2 read of a digest written by another CTA in this launch.
__device__ __forceinline__ void ld_dig_cg(const uint64_t* p, uint64_t (&d)[4]) {
  ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2*>(p));
  ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2*>(p) + 1);
  d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
}

// This thread's warp, as a value the compiler knows to be the same in all of the
// warp's lanes.
__device__ __forceinline__ uint32_t warp_index() { return __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); }

template <uint32_t KIND>
__device__ __forceinline__ void leaf_digest(const TreeJob& job, uint64_t leaf, const uint32_t (&ch)[4], uint64_t (&d)[4]) {
  if constexpr (KIND == kLeafQM31) {
    uint4 v = ld_written(job.layer + leaf);
    sha3_16((uint64_t)v.x | ((uint64_t)v.y << 32), (uint64_t)v.z | ((uint64_t)v.w << 32), d);
  } else if constexpr (KIND == kLeafDigest) {
    ld_dig(reinterpret_cast<const uint64_t*>(job.raw) + 4 * leaf, d);
  } else {
    hash_message<true>(job.raw + leaf * job.stride, job.len, job.suffix, job.aligned8 != 0, d);
  }
}

// The challenge of a fold kind, read by every thread beside its first values: through
// shared memory and a barrier ahead of them it cost each round 400 to 750 cycles.
template <uint32_t KIND>
__device__ __forceinline__ void fold_challenge(const TreeJob& job, uint32_t (&ch)[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) ch[k] = KIND == kLeafFold || KIND == kLeafFoldx4 || KIND == kLeafFoldQ ? __ldcg(job.fold_ch + k) : 0u;
}

// Value e of the layer that a fold kind produces.
template <uint32_t KIND>
__device__ __forceinline__ uint4 folded_value(const TreeJob& job, uint64_t e, const uint32_t (&ch)[4]) {
  const uint4 p = ld_written(job.layer + 2 * e), q = ld_written(job.layer + 2 * e + 1);
  const qm31 pos = {p.x, p.y, p.z, p.w}, neg = {q.x, q.y, q.z, q.w}, c = {ch[0], ch[1], ch[2], ch[3]};
  qm31 r;
  if constexpr (KIND == kLeafFoldQ) {
    const uint4 t = __ldg(reinterpret_cast<const uint4*>(job.inv) + e);
    r = fri_fold_pair_q(pos, neg, qm31{t.x, t.y, t.z, t.w}, c);
  } else {
    r = fri_fold_pair(pos, neg, __ldg(job.inv + e), c);
  }
  return make_uint4(r.a, r.b, r.c, r.d);
}

// A raw message and its suffix into the first LANES (9, messages below 72 bytes, or
// 17) of a zero state.  A compare, a select and an XOR for each lane of the rate took
// 0.5 % of a tree of 2^22 64-byte leaves.
template <uint32_t LANES>
__device__ __forceinline__ void raw_setup(const TreeJob& job, uint64_t leaf, uint64_t (&a)[25]) {
  const uint8_t* const p = job.raw + leaf * job.stride;
  const uint32_t full = job.len >> 3, rem = job.len & 7;
  uint64_t tail = (uint64_t)job.suffix << (8 * rem);
  if (job.aligned8) {
    if (rem) tail |= aligned_tail(p + 8 * full, rem);
#pragma unroll
    for (uint32_t i = 0; i < LANES; i++)
      if (i < full) a[i] = __ldg(reinterpret_cast<const uint64_t*>(p) + i);
  } else {
    // 2^20 leaves of 99 bytes: 606 us, 598 with whole units; 618 with both readers in this
    // loop's code, one for the first and last leaf
    const UnalignedWords<true> u(p, job.len);
    if (rem) tail |= u.word(full, rem);
#pragma unroll
    for (uint32_t i = 0; i < LANES; i++)
      if (i < full) a[i] = u.word(i, 8);
  }
#pragma unroll
  for (uint32_t i = 0; i < LANES; i++)
    if (i == full) a[i] = tail;
}

// Sets up the sponge input of one leaf (message lanes, suffix and end padding)
// and returns how many permutations it takes (2 for a 136-byte raw leaf).
template <uint32_t KIND>
__device__ __forceinline__ uint32_t leaf_setup(const TreeJob& job, uint64_t leaf, const uint32_t (&ch)[4], uint64_t (&a)[25]) {
  if constexpr (KIND == kLeafQM31x4 || KIND == kLeafFoldx4) {
    // leaf = values 4*leaf .. 4*leaf+3 (64 bytes, 8 lanes)
#pragma unroll
    for (uint32_t m = 0; m < 4; m++) {
      const uint64_t e = 4 * leaf + m;
      uint4 v;
      if constexpr (KIND == kLeafQM31x4) {
        v = ld_written(job.layer + e);
      } else {
        v = folded_value<KIND>(job, e, ch);
        job.out_layer[e] = v;
      }
      a[2 * m] = (uint64_t)v.x | ((uint64_t)v.y << 32);
      a[2 * m + 1] = (uint64_t)v.z | ((uint64_t)v.w << 32);
    }
    a[8] = 0x06;
    a[16] = kPadEnd;
    return 1;
  } else {
    if (job.len < 72) raw_setup<9>(job, leaf, a);
    else raw_setup<17>(job, leaf, a);
    if (job.len == 136) return 2;
    a[16] ^= kPadEnd;
    return 1;
  }
}

// ---------------------------------------------------------------------------
// Shared digest buffers.  A buffer of more than kStdDigests digests holds them
// split into even and odd bits (two 16-byte words each, the form a pair of lanes
// hashes); smaller ones hold them as they are (four u64 lanes), for the levels that
// take a warp per node.
// ---------------------------------------------------------------------------
static constexpr uint32_t kStdLog = 3, kStdDigests = 1u << kStdLog;
// Digests that the leaf phase of a 2^tl-leaf treelet leaves in shared memory, and
// the height of the subtree each thread hashed: with fewer than THREADS leaves a
// pair of lanes takes each leaf (latency is all there is), with fewer than
// 4 x THREADS each thread hashes one or two leaves, else a 4-leaf subtree.  A small
// tree is a chain of dependent permutations, so what bounds it is their latency
// (4.5 us by a thread, 2.75 us by a pair, 2.2 us by a warp, at 1.965 GHz); a large
// one is bound by integer issue, where a thread per subtree is 2 to 7 % better than
// pairs.  With every level by threads, the 2^10-leaf commit took 116 us a call, a
// 2^16-value commit-and-fold chain of 10 rounds 1263 us and a 2^22 proof 8090 us;
// with this split 70, 745 and 7310 us.
__host__ __device__ constexpr uint32_t tree_subtree_height(uint32_t leaves, uint32_t threads) {
  return leaves >= 4 * threads ? 2u : leaves >= 2 * threads ? 1u : 0u;
}
__host__ __device__ constexpr uint32_t tree_phase_digests(uint32_t leaves, uint32_t threads) {
  const uint32_t m = leaves >> tree_subtree_height(leaves, threads);
  return m < kStdDigests ? kStdDigests : m;
}
// The last levels' digests: up to kStdDigests of them, then each level behind the
// one below it.
static constexpr uint32_t kTopWords = 4 * (2 * kStdDigests);
// Dynamic shared memory of a launch whose deepest treelet has 2^tl leaves: the
// leaf phase's digests and half as many for the level above.  Shallower treelets of
// the same launch need no more than max(12 bytes per leaf, 48 x threads).
static size_t tree_smem_bytes(uint32_t max_tile_log, uint32_t threads) {
  const uint32_t leaves = 1u << max_tile_log;
  size_t m = tree_phase_digests(leaves, threads);
  if (leaves > threads && m < threads) m = threads;
  return 48 * m;
}

// Leaf phase by threads: subtrees of height h = 0, 1 or 2, one per thread.  Items
// are the tile's leaves.  The subtree's inner nodes are stored (levels 1 .. h,
// first node idx0 >> l) and its root written to `out` in shared memory.  A 4-leaf
// subtree runs as a 7-step loop around ONE permutation site (leaf, leaf, pair,
// leaf, leaf, pair, pair), which keeps the kernel's code small enough for the
// instruction cache.
template <uint32_t KIND, int THREADS>
__device__ __noinline__ void subtree_phase(const TreeJob& job, uint32_t items, uint32_t h, uint64_t idx0, uint64_t* out) {
  uint32_t ch[4];
  fold_challenge<KIND>(job, ch);
  const uint32_t groups = items >> h;
  const uint64_t* digests = reinterpret_cast<const uint64_t*>(job.raw) + 4 * idx0;
  uint64_t* l1 = job.inner + 4 * (inner_offset(job.logn, 1) + (idx0 >> 1));
  uint64_t* l2 = job.inner + 4 * (inner_offset(job.logn, 2) + (idx0 >> 2));
  // step k: item index within the subtree (leaf steps) and the step's kind
  //   k:     0  1  2  3  4  5  6        (h == 2)
  //   item:  0  1  -  2  3  -  -
  const uint32_t steps = h == 2 ? 7 : (h == 1 ? 3 : 1);
  for (uint32_t j = threadIdx.x; j < groups; j += THREADS) {
    // A pair's right child is always the digest of the step before it; its left child
    // waits in this thread's place of `out` (a leaf) or in the level it was stored to
    // (the first pair): the memory pipe is idle, while carrying both in registers and
    // selecting per step cost the integer pipe 1 % of all its instructions.
    ulonglong2* const mine = reinterpret_cast<ulonglong2*>(out) + 2 * j;
    uint64_t d[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (uint32_t k = 0; k < steps; k++) {
      const bool pair = (h == 2) ? (k == 2 || k == 5 || k == 6) : (h == 1 && k == 2);
      const uint32_t item = k < 2 ? k : k - 1;  // leaf steps only (h == 2: k = 0, 1, 3, 4)
      const uint64_t leaf = idx0 + (uint64_t)j * (1u << h) + item;
      if (!pair && KIND == kLeafDigest) {
        ld_dig_cg(digests + 4 * ((uint64_t)j * (1u << h) + item), d);
      } else {
        uint64_t a[25];
#pragma unroll
        for (int i = 0; i < 17; i++) a[i] = 0;
        if (pair) {
          const ulonglong2* const l = k == 6 ? reinterpret_cast<const ulonglong2*>(l1 + 8 * j) : mine;
          const ulonglong2 l0 = l[0], l1v = l[1];
          a[0] = l0.x, a[1] = l0.y, a[2] = l1v.x, a[3] = l1v.y;
#pragma unroll
          for (int i = 0; i < 4; i++) a[4 + i] = d[i];
          a[8] = 0x06;
          a[16] = kPadEnd;
        } else if (leaf_setup<KIND>(job, leaf, ch, a) == 2) {  // a full block, then the padding's own
#pragma unroll
          for (int i = 17; i < 25; i++) a[i] = 0;
          keccak_f1600(a);
          a[0] ^= job.suffix;
          a[16] ^= kPadEnd;
          keccak_digest<kLanesAll>(a, d);
          goto hashed;
        }
        keccak_digest<KIND == kLeafRaw ? kLanesRate : kLanes64>(a, d);
      hashed:
        if (!pair && job.leaf_digests) st_dig(job.leaf_digests + 4 * leaf, d);
      }
      if (steps > 1 && (k == 0 || k == 3)) mine[0] = make_ulonglong2(d[0], d[1]), mine[1] = make_ulonglong2(d[2], d[3]);
      if (h == 2 && k == 2) st_dig(l1 + 8 * j, d);
      if (h == 2 && k == 5) st_dig(l1 + 8 * j + 4, d);
      if (h == 2 && k == 6) st_dig(l2 + 4 * j, d);
      if (h == 1 && k == 2) st_dig(l1 + 4 * j, d);
      if (k + 1 == steps) {
        // at least THREADS digests, more than kStdDigests: split form
        uint4 e, o;
        split64(d[0], e.x, o.x);
        split64(d[1], e.y, o.y);
        split64(d[2], e.z, o.z);
        split64(d[3], e.w, o.w);
        reinterpret_cast<uint4*>(out)[2 * j] = e;
        reinterpret_cast<uint4*>(out)[2 * j + 1] = o;
      }
    }
  }
  __syncthreads();
}

// The same for leaves of one 16-byte value, in split form throughout: a value's two
// lanes are split, the inner nodes joined for their store.  The first pair's digest
// waits, split, in the place of the level-2 node that this thread stores at the end.
// Per permutation of a 2^22-value tree 4178 integer instructions (4261 unsplit), 2073 ->
// 2017 us; a fold's tree of 2^21 1105 -> 1067 us.  Longer leaves would lose the 6
// instructions a round again to splitting their words.
template <uint32_t KIND, int THREADS>
__device__ __noinline__ void value_subtree_phase(const TreeJob& job, uint32_t items, uint32_t h, uint64_t idx0, uint64_t* out) {
  uint32_t ch[4];
  fold_challenge<KIND>(job, ch);
  const uint32_t groups = items >> h, steps = h == 2 ? 7 : (h == 1 ? 3 : 1);
  uint64_t* l1 = job.inner + 4 * (inner_offset(job.logn, 1) + (idx0 >> 1));
  uint64_t* l2 = job.inner + 4 * (inner_offset(job.logn, 2) + (idx0 >> 2));
  for (uint32_t j = threadIdx.x; j < groups; j += THREADS) {
    SplitDigest* const mine = reinterpret_cast<SplitDigest*>(out) + j;
    SplitDigest* const first = reinterpret_cast<SplitDigest*>(l2 + 4 * j);
    SplitDigest d = {};
#pragma unroll 1
    for (uint32_t k = 0; k < steps; k++) {
      const bool pair = h == 2 ? (k == 2 || k == 5 || k == 6) : k == 2;
      const uint32_t item = k < 2 ? k : k - 1;  // leaf steps only
      const uint64_t leaf = idx0 + (uint64_t)j * (1u << h) + item;
      uint32_t e[25], o[25];
      e[16] = 0, o[16] = 0x80000000u;  // the end padding
      if (pair) {
        const SplitDigest l = k == 6 ? *first : *mine;
        e[0] = l.even.x, e[1] = l.even.y, e[2] = l.even.z, e[3] = l.even.w;
        o[0] = l.odd.x, o[1] = l.odd.y, o[2] = l.odd.z, o[3] = l.odd.w;
        e[4] = d.even.x, e[5] = d.even.y, e[6] = d.even.z, e[7] = d.even.w;
        o[4] = d.odd.x, o[5] = d.odd.y, o[6] = d.odd.z, o[7] = d.odd.w;
        e[8] = 2, o[8] = 1;  // 0x06
        split_round<kLanes64>(e, o, 0);
      } else {
        uint4 v;
        if constexpr (KIND == kLeafQM31) {
          v = ld_written(job.layer + leaf);
        } else {
          v = folded_value<KIND>(job, leaf, ch);
          job.out_layer[leaf] = v;
        }
        split64((uint64_t)v.x | ((uint64_t)v.y << 32), e[0], o[0]);
        split64((uint64_t)v.z | ((uint64_t)v.w << 32), e[1], o[1]);
        e[2] = 2, o[2] = 1;
        split_round<kLanes16>(e, o, 0);
      }
      d = split_digest_rest(e, o);
      uint64_t* node = nullptr;
      if (!pair) node = job.leaf_digests ? job.leaf_digests + 4 * leaf : nullptr;
      else if (k == 6) node = l2 + 4 * j;
      else node = l1 + (h == 2 ? 8 * j + (k == 5 ? 4 : 0) : 4 * j);
      if (node) {
        const uint64_t w[4] = {join64(d.even.x, d.odd.x), join64(d.even.y, d.odd.y), join64(d.even.z, d.odd.z), join64(d.even.w, d.odd.w)};
        st_dig(node, w);
      }
      if (k + 1 == steps || k == 0 || k == 3) *mine = d;
      else if (k == 2) *first = d;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ ulonglong2 pack_qm31(uint4 v) {
  return make_ulonglong2((uint64_t)v.x | ((uint64_t)v.y << 32), (uint64_t)v.z | ((uint64_t)v.w << 32));
}
// Word i of a raw message with its suffix (none at length 136); word(i, n): its n
// bytes.
template <class F>
__device__ __forceinline__ uint64_t raw_message_word(const TreeJob& job, uint32_t i, F word) {
  const uint32_t full = job.len >> 3, rem = job.len & 7;
  if (i > full || i > 16) return 0;
  const uint32_t n = i < full ? 8 : rem;
  const uint64_t v = i < full ? 0 : (uint64_t)job.suffix << (8 * rem);
  return n ? v | word(i, n) : v;
}

// Digest of one leaf by a pair of lanes, in split form.  `ok`: the pair's leaf is
// inside the tile (its stores happen).
template <uint32_t KIND>
__device__ __forceinline__ uint4 pair_leaf(const TreeJob& job, uint64_t leaf, bool ok, const uint32_t (&ch)[4], uint32_t q) {
  if constexpr (KIND == kLeafDigest) {
    return pair_split_digest(__ldcg(reinterpret_cast<const ulonglong2*>(job.raw) + 2 * leaf + q), q);
  } else {
    uint32_t a[25];
#pragma unroll
    for (int i = 0; i < 25; i++) a[i] = 0;
    if constexpr (KIND == kLeafQM31 || KIND == kLeafFold || KIND == kLeafFoldQ) {
      uint4 v;
      if constexpr (KIND == kLeafQM31) {
        v = ld_written(job.layer + leaf);
      } else {
        v = folded_value<KIND>(job, leaf, ch);
        if (ok && q == 0) job.out_layer[leaf] = v;
      }
      const ulonglong2 w = pack_qm31(v);
      pair_split2(q ? w.y : w.x, q, a[0], a[1]);
      a[2] = pair_suffix(0x06, q);
    } else if constexpr (KIND == kLeafQM31x4 || KIND == kLeafFoldx4) {
      // thread q takes values 2q and 2q + 1 (lanes 4q .. 4q + 3)
#pragma unroll
      for (uint32_t m = 0; m < 2; m++) {
        const uint64_t e = 4 * leaf + 2 * q + m;
        uint4 v;
        if constexpr (KIND == kLeafQM31x4) {
          v = ld_written(job.layer + e);
        } else {
          v = folded_value<KIND>(job, e, ch);
          if (ok) job.out_layer[e] = v;
        }
        const ulonglong2 w = pack_qm31(v);
        pair_split2(w.x, q, a[2 * m], a[4 + 2 * m]);
        pair_split2(w.y, q, a[2 * m + 1], a[5 + 2 * m]);
      }
      a[8] = pair_suffix(0x06, q);
    } else {
      // words 2m by thread 0, 2m + 1 by thread 1
      const uint8_t* p = job.raw + leaf * job.stride;
      auto words = [&](auto word) {
        const uint32_t last = job.len >> 3;
#pragma unroll
        for (uint32_t m = 0; m < 9; m++) {
          if (2 * m > last) continue;  // the same for the whole launch
          uint32_t w1;
          pair_split2(raw_message_word(job, 2 * m + q, word), q, a[2 * m], w1);
          if (m < 8) a[2 * m + 1] = w1;
        }
      };
      if (job.aligned8) {
        words([&](uint32_t i, uint32_t n) { return n == 8 ? __ldg(reinterpret_cast<const uint64_t*>(p) + i) : aligned_tail(p + 8 * i, n); });
      } else {
        const UnalignedWords<true> u(p, job.len);
        words([&](uint32_t i, uint32_t n) { return u.word(i, n); });
      }
    }
    if (KIND == kLeafRaw && job.len == 136) {  // a full block, then the padding's own
      pair_f1600(a, q);
      a[0] ^= pair_suffix(job.suffix, q);
      a[16] ^= pair_pad_end(q);
      return pair_digest<kLanesAll>(a, q);
    }
    a[16] ^= pair_pad_end(q);
    return pair_digest<KIND == kLeafRaw ? kLanesRate : KIND == kLeafQM31x4 || KIND == kLeafFoldx4 ? kLanes64 : kLanes16>(a, q);
  }
}

// Digest i of `count` into shared memory (`buf` in split form, or `top` as it is)
// and, joined, to global memory (`node`, null for none).
__device__ __forceinline__ void put_digest(uint64_t* buf, uint64_t* top, uint32_t count, uint32_t i, uint4 d, uint64_t* node, bool ok, uint32_t q) {
  const bool std_form = count <= kStdDigests;
  if (node != nullptr || std_form) {  // the same for the whole warp
    const ulonglong2 j = pair_join_digest(d, q);
    if (ok && node != nullptr) reinterpret_cast<ulonglong2*>(node)[q] = j;
    if (ok && std_form) reinterpret_cast<ulonglong2*>(top)[2 * i + q] = j;
  }
  if (ok && !std_form) reinterpret_cast<uint4*>(buf)[2 * i + q] = d;
}

// Leaf phase by pairs of lanes (fewer leaves than threads).
template <uint32_t KIND, int THREADS>
__device__ __noinline__ void pair_leaf_phase(const TreeJob& job, uint32_t items, uint64_t idx0, uint64_t* out, uint64_t* top) {
  uint32_t ch[4];
  fold_challenge<KIND>(job, ch);
  const uint32_t lane = threadIdx.x & 31, q = lane & 1;
  for (uint32_t base = warp_index() * 16; base < items; base += THREADS / 2) {
    const uint32_t i = base + (lane >> 1);
    const bool ok = i < items;
    const uint64_t leaf = idx0 + (ok ? i : items - 1);
    const uint4 d = pair_leaf<KIND>(job, leaf, ok, ch, q);
    put_digest(out, top, items, i, d, job.leaf_digests ? job.leaf_digests + 4 * leaf : nullptr, ok, q);
  }
  __syncthreads();
}

// Levels of at least kStdDigests nodes, a pair of lanes per node, until kStdDigests
// digests are left (in `top`): from `count` digests in buffer `a` (scratch `b`), or
// (nodes != null) from the `count` tree nodes at `nodes`, written by other CTAs.
// `level`, `idx0`: level and first node index of the digests; both advance.
template <int THREADS>
__device__ __noinline__ void pair_levels(uint64_t* a, uint64_t* b, uint64_t* top, const uint64_t* nodes, uint32_t n, const TreeJob& job, uint32_t level,
                                         uint64_t idx0) {
  const uint32_t warp = warp_index(), lane = threadIdx.x & 31, q = lane & 1;
  uint64_t* src = a;
  uint64_t* dst = b;
  if (nodes != nullptr) dst = a;
  while (n > kStdDigests) {
    n >>= 1;
    idx0 >>= 1;
    level++;
    uint64_t* lv = job.inner + 4 * (inner_offset(job.logn, level) + idx0);
    for (uint32_t base = warp * 16; base < n; base += THREADS / 2) {
      const uint32_t i = base + (lane >> 1);
      const bool ok = i < n;
      const uint32_t j = ok ? i : n - 1;
      uint4 l, r;
      if (nodes != nullptr) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(nodes) + 4 * j + q;
        l = pair_split_digest(__ldcg(p), q);
        r = pair_split_digest(__ldcg(p + 2), q);
      } else {
        const uint4* p = reinterpret_cast<const uint4*>(src) + 4 * j + q;
        l = p[0];
        r = p[2];
      }
      put_digest(dst, top, n, i, pair_hash_parent(l, r, q), lv + 4 * j, ok, q);
    }
    __syncthreads();
    if (nodes != nullptr) {
      nodes = nullptr;
      src = dst;
      dst = b;
    } else {
      uint64_t* t = src;
      src = dst;
      dst = t;
    }
  }
}

// The last levels (at most kStdDigests digests in `top`) with a warp per node, and
// in the CTA that reaches the root the root's transcript round.  The transcript's
// first absorptions (the public digest before round 0, the commitment frame) need
// no root, so the fourth warp takes them while the first two hash the top nodes.
template <int THREADS>
__device__ __noinline__ void top_levels(uint64_t* top, uint32_t count, const TreeJob& job, uint32_t level, uint64_t idx0, bool root, uint64_t* warp_smem) {
  static_assert(THREADS >= 128, "four warps");
  const uint32_t warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t act = root ? job.root_action : (uint32_t)kRootNone;
  if (warp >= 4) return;
  if (warp == 3 && act != kRootNone) {
    // one permutation site for all of this warp's steps
    enum { kNode, kPublic, kCommit, kRoot, kChallenge };
    WarpSponge sp(warp_smem + kWarpKeccakWords * 3);
    sp.load(job.base ? job.base : job.transcript);
    const uint64_t state = sp.a;
    RoundFrames f = {0, 0};
    uint64_t* const node = top + 8 * 4 + 4 * 3;  // the fourth node above eight digests
    // the node that the other warps wait for first: the state's load and the frames
    // ahead of it held the level above eight digests up by 1000 cycles (with the fold
    // challenge, chain of 10 trees 537 -> 533 us, 2^10 opening 258 -> 252)
#pragma unroll 1
    for (uint32_t step = count == 8 ? kNode : kPublic; step <= kChallenge; step++) {
      uint64_t word = 0;
      if (step == kNode) {
        sp.a = lane < 8 ? top[24 + lane] : lane == 8 ? 0x06ull : lane == 16 ? kPadEnd : 0ull;
      } else if (step == kPublic) {
        if (!job.pub) continue;
        word = sp.digest_word(job.pub);
      } else if (step == kCommit) {
        f = act == kRootCircleRound ? circle_round_frames(lane, job.round) : qm31_round_frames(lane, job.round, job.frame_in_count);
        word = f.commit;
      } else if (step == kRoot) {
        asm volatile("bar.sync 2, 128;" ::: "memory");
        word = sp.digest_word(top + (count == 8 ? 56 : count == 4 ? 24 : count == 2 ? 8 : 0));
      } else {
        word = f.challenge;
      }
      sp.absorb(word);
      if (step == kNode) {
        uint64_t* const out = job.inner + 4 * (inner_offset(job.logn, level + 1) + (idx0 >> 1) + 3);
        if (lane < 4) node[lane] = out[lane] = sp.a;
        sp.a = state;
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
    }
    uint32_t ch[4];
    sp.squeeze4_m31(ch);
    sp.store(job.transcript);
    if (lane == 0)
      for (int k = 0; k < 4; k++) job.challenge_out[k] = ch[k];
    return;
  }
  const WarpKeccak kf(lane, warp_smem + kWarpKeccakWords * warp);
  uint64_t* src = top;
  uint32_t n = count;
  while (n > 1) {
    n >>= 1;
    idx0 >>= 1;
    level++;
    uint64_t* const dst = src + 8 * n;
    if (warp < n) {
      uint64_t* const node = job.inner + 4 * (inner_offset(job.logn, level) + idx0 + warp);
      uint64_t a = lane < 8 ? src[8 * warp + lane] : lane == 8 ? 0x06ull : lane == 16 ? kPadEnd : 0ull;
      kf.permute_small(a);
      if (lane < 4) dst[4 * warp + lane] = node[lane] = a;
    }
    // four nodes take all four warps; below that only the first two go on
    if (n == 4) {
      asm volatile("bar.sync 1, 128;" ::: "memory");
    } else if (n == 2) {
      if (warp >= 2) break;
      asm volatile("bar.sync 3, 64;" ::: "memory");
    }
    src = dst;
  }
  if (root && warp == 0 && lane < 4 && job.root_out) job.root_out[lane] = src[lane];
  if (act != kRootNone) asm volatile("bar.sync 2, 128;" ::: "memory");
}

// One tile of one job: leaf digests, treelet, then the last-arriver climb.
template <uint32_t KIND, int THREADS>
__device__ __forceinline__ void tree_tile_body(const TreeJob& job, const uint64_t tile) {
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ __align__(16) uint64_t warp_smem[4 * kWarpKeccakWords];
  __shared__ __align__(16) uint64_t top[kTopWords];
  __shared__ uint32_t s_last;
  const uint32_t tl = job.tile_log < job.logn ? job.tile_log : job.logn;
  const uint32_t T = 1u << tl;
  const uint32_t M = tree_phase_digests(T, THREADS);  // capacity of bufA; bufB holds half
  uint64_t* bufA = sm;
  uint64_t* bufB = sm + 4 * M;

  // 1) leaf digests (and the lowest levels of this tile, per thread)
  const uint64_t first = tile * T;
  uint32_t h = 0;
  if (T < THREADS) {
    pair_leaf_phase<KIND, THREADS>(job, T, first, bufA, top);
  } else {
    h = tree_subtree_height(T, THREADS);
    if constexpr (KIND == kLeafQM31 || KIND == kLeafFold || KIND == kLeafFoldQ)
      value_subtree_phase<KIND, THREADS>(job, T, h, first, bufA);
    else
      subtree_phase<KIND, THREADS>(job, T, h, first, bufA);
  }
  // 2) treelet: the levels above, to kStdDigests digests and then to the root
  uint32_t top_log = tl < kStdLog ? tl : kStdLog;
  pair_levels<THREADS>(bufA, bufB, top, nullptr, T >> h, job, h, first >> h);
  top_levels<THREADS>(top, 1u << top_log, job, tl - top_log, first >> (tl - top_log), tl == job.logn, warp_smem);
  // 3) climb: last arriver of each group continues
  uint32_t level = tl;
  uint64_t idx = tile;
  uint64_t cnt_off = 0;
  while (level < job.logn) {
    uint32_t glog = job.group_log;
    if (glog > job.logn - level) glog = job.logn - level;
    while (glog > 1 && (1u << glog) > 2 * M) glog--;  // the group's first level must fit bufA
    const uint32_t G = 1u << glog;
    const uint64_t gidx = idx >> glog;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      uint32_t old = atomicAdd(job.counters + cnt_off + gidx, 1u);
      s_last = (old == G - 1) ? 1u : 0u;
      if (s_last) job.counters[cnt_off + gidx] = 0;  // reset for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint64_t* lv = job.inner + 4 * (inner_offset(job.logn, level) + gidx * G);
    top_log = glog < kStdLog ? glog : kStdLog;
    if (G > kStdDigests) {
      pair_levels<THREADS>(bufA, bufB, top, lv, G, job, level, gidx * G);
    } else {
      if (threadIdx.x < 4 * G) top[threadIdx.x] = __ldcg(lv + threadIdx.x);
      __syncthreads();
    }
    const uint32_t up = level + glog - top_log;
    top_levels<THREADS>(top, 1u << top_log, job, up, (gidx * G) >> (glog - top_log), level + glog == job.logn, warp_smem);
    cnt_off += (1ull << (job.logn - level)) >> glog;
    level += glog;
    idx = gidx;
  }
}

// The job in shared memory: read once per CTA, not by every use in turn.
__device__ __forceinline__ void fetch_job(TreeJob& to, const TreeJob* from) {
  static_assert(sizeof(TreeJob) % 8 == 0, "whole words");
  if (threadIdx.x < sizeof(TreeJob) / 8) reinterpret_cast<uint64_t*>(&to)[threadIdx.x] = __ldg(reinterpret_cast<const uint64_t*>(from) + threadIdx.x);
  __syncthreads();
}

template <uint32_t KIND, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) tree_tiles_kernel(const TreeJob* __restrict__ jobs, const uint2* __restrict__ work) {
  __shared__ TreeJob job;
  const uint2 w = work[blockIdx.x];
  fetch_job(job, jobs + w.x);
  // Launched before the kernel ahead of it in the stream has ended (launch_kind): up
  // to here only the work list and the job were read, which no kernel writes; layers,
  // challenge, transcript, nodes and counters are touched once that kernel's memory is
  // complete.
  dependent_begin();
  tree_tile_body<KIND, THREADS>(job, w.y);
}

// Persistent form: a grid of the resident CTAs pulls work items from a device
// counter (queue[0]) until the list is done.  Nothing waits on anything: the
// last-arriver climb is unchanged, and the last CTA to leave (queue[1] counts
// them) resets both counters, so a captured launch sequence replays.
template <uint32_t KIND, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) tree_queue_kernel(const TreeJob* __restrict__ jobs, const uint2* __restrict__ work,
                                                                            uint32_t nwork, uint32_t* __restrict__ queue) {
  __shared__ uint32_t s_item;
  __shared__ TreeJob job;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
    __syncthreads();
    const uint32_t item = s_item;
    __syncthreads();  // every thread has the item (and the last one's shared memory is free)
    if (item >= nwork) break;
    const uint2 w = work[item];
    fetch_job(job, jobs + w.x);
    tree_tile_body<KIND, THREADS>(job, w.y);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(queue + 1, 1u) == gridDim.x - 1) {
      queue[0] = 0;
      queue[1] = 0;
    }
  }
}

// Single job passed by value, tile = blockIdx.x: needs no job or work-list buffer.
template <uint32_t KIND, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) tree_direct_kernel(const TreeJob job) {
  tree_tile_body<KIND, THREADS>(job, blockIdx.x);
}

static constexpr int kMaxTreeLog = 13;
static constexpr int kMaxTreeSmem = 12 << kMaxTreeLog;  // 2^11 digests + 2^10 digests (48 x 512 threads is less)

template <uint32_t KIND>
static cudaError_t prepare_kind() {
  cudaError_t e = cudaSuccess;
  for (auto k : {tree_tiles_kernel<KIND, 128>, tree_tiles_kernel<KIND, 256>, tree_tiles_kernel<KIND, 512>}) {
    cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTreeSmem);
    if (r != cudaSuccess) e = r;
  }
  for (auto k : {tree_queue_kernel<KIND, 128>, tree_queue_kernel<KIND, 256>, tree_queue_kernel<KIND, 512>}) {
    cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTreeSmem);
    if (r != cudaSuccess) e = r;
  }
  return e;
}

// Opt the tree kernels into > 48 KiB of dynamic shared memory once, outside any
// stream capture.
cudaError_t prepare_tree_kernels() {
  cudaError_t e = prepare_kind<kLeafRaw>();
  if (e == cudaSuccess) e = prepare_kind<kLeafQM31>();
  if (e == cudaSuccess) e = prepare_kind<kLeafFold>();
  if (e == cudaSuccess) e = prepare_kind<kLeafDigest>();
  if (e == cudaSuccess) e = prepare_kind<kLeafQM31x4>();
  if (e == cudaSuccess) e = prepare_kind<kLeafFoldx4>();
  if (e == cudaSuccess) e = prepare_kind<kLeafFoldQ>();
  return e;
}

// Resident CTAs of a persistent launch: the occupancy of the kernel at this
// shared-memory size times the SMs, no more than the work items.
template <class K>
static uint32_t resident_grid(K kernel, int threads, size_t smem, uint32_t nwork) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
    if (sms < 1) sms = 148;
  }
  const uint64_t g = (uint64_t)sms * (uint64_t)per_sm;
  return (uint32_t)(g < nwork ? g : nwork);
}

template <uint32_t KIND>
static cudaError_t launch_kind(const TreeJob* d_jobs, const uint2* d_work, uint32_t nwork, uint32_t max_tile_log, uint32_t threads, uint32_t* queue,
                               cudaStream_t s) {
  const size_t smem = tree_smem_bytes(max_tile_log, threads == 128 || threads == 512 ? threads : 256);
  if (queue) {
    if (threads == 128)
      tree_queue_kernel<KIND, 128><<<resident_grid(tree_queue_kernel<KIND, 128>, 128, smem, nwork), 128, smem, s>>>(d_jobs, d_work, nwork, queue);
    else if (threads == 512)
      tree_queue_kernel<KIND, 512><<<resident_grid(tree_queue_kernel<KIND, 512>, 512, smem, nwork), 512, smem, s>>>(d_jobs, d_work, nwork, queue);
    else
      tree_queue_kernel<KIND, 256><<<resident_grid(tree_queue_kernel<KIND, 256>, 256, smem, nwork), 256, smem, s>>>(d_jobs, d_work, nwork, queue);
    return cudaGetLastError();
  }
  // the commit launches of a fold chain follow one another, each ending in the last
  // arriver's climb with most SMs idle
  if (threads == 128) return launch_dependent(tree_tiles_kernel<KIND, 128>, dim3(nwork), dim3(128), smem, s, d_jobs, d_work);
  if (threads == 512) return launch_dependent(tree_tiles_kernel<KIND, 512>, dim3(nwork), dim3(512), smem, s, d_jobs, d_work);
  return launch_dependent(tree_tiles_kernel<KIND, 256>, dim3(nwork), dim3(256), smem, s, d_jobs, d_work);
}

cudaError_t launch_tree_jobs(const TreeJob* d_jobs, const uint2* d_work, uint32_t nwork, uint32_t max_tile_log, uint32_t kind, uint32_t threads,
                             cudaStream_t s, uint32_t* d_queue) {
  if (nwork == 0) return cudaSuccess;
  if (max_tile_log > kMaxTreeLog) return cudaErrorInvalidValue;
  switch (kind) {
    case kLeafRaw: return launch_kind<kLeafRaw>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafQM31: return launch_kind<kLeafQM31>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafFold: return launch_kind<kLeafFold>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafDigest: return launch_kind<kLeafDigest>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafQM31x4: return launch_kind<kLeafQM31x4>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafFoldx4: return launch_kind<kLeafFoldx4>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    case kLeafFoldQ: return launch_kind<kLeafFoldQ>(d_jobs, d_work, nwork, max_tile_log, threads, d_queue, s);
    default: return cudaErrorInvalidValue;
  }
}

// One raw-leaf tree, job by value, 256 threads, treelets of at most 2^9 leaves
// (12 KiB of dynamic shared memory: under the default limit, no opt-in needed).
cudaError_t launch_tree_direct_raw(const TreeJob& job, cudaStream_t s) {
  if (job.tile_log > 9 || (job.logn > 0 && job.tile_log == 0)) return cudaErrorInvalidValue;
  uint32_t tl = job.tile_log < job.logn ? job.tile_log : job.logn;
  unsigned tiles = 1u << (job.logn - tl);
  tree_direct_kernel<kLeafRaw, 256><<<tiles, 256, tree_smem_bytes(tl, 256), s>>>(job);
  return cudaGetLastError();
}

// Sibling paths for leaves of a committed tree: out[k][level] = digest of the
// sibling at `level` (bottom-up), depth = job.logn digests per index.  Level 0
// comes from stored leaf digests, or is recomputed from the leaf source.
__global__ void gather_openings_kernel(const TreeJob* __restrict__ jobp, const uint64_t* __restrict__ idx, uint32_t nidx, uint64_t* __restrict__ out) {
  const TreeJob& job = *jobp;
  uint32_t depth = job.logn;
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (uint64_t)nidx * depth) return;
  uint32_t k = (uint32_t)(t / depth), level = (uint32_t)(t % depth);
  uint64_t leaf = idx[k];
  uint64_t node = (leaf >> level) ^ 1ull;
  uint64_t d[4];
  if (level == 0) {
    if (job.leaf_digests) {
      ld_dig(job.leaf_digests + 4 * node, d);
    } else {
      uint32_t ch[4] = {0, 0, 0, 0};
      if (job.kind == kLeafQM31)
        leaf_digest<kLeafQM31>(job, node, ch, d);
      else if (job.kind == kLeafDigest)
        leaf_digest<kLeafDigest>(job, node, ch, d);
      else
        leaf_digest<kLeafRaw>(job, node, ch, d);
    }
  } else {
    ld_dig(job.inner + 4 * (inner_offset(job.logn, level) + node), d);
  }
  st_dig(out + 4 * ((uint64_t)k * depth + level), d);
}

cudaError_t launch_gather_openings(const TreeJob* d_job, const uint64_t* d_idx, uint32_t nidx, uint64_t* d_out, cudaStream_t s) {
  // depth is read on the device; launch enough threads for the deepest tree (31 levels)
  uint64_t total = (uint64_t)nidx * 32;
  if (total == 0) return cudaSuccess;
  gather_openings_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_job, d_idx, nidx, d_out);
  return cudaGetLastError();
}

}  // namespace azk

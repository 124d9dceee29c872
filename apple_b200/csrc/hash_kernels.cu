// Batch Keccak-f[1600] permutations and fixed-rate SHA3-256 / Keccak-256 batch
// hashing (KeccakF1600PermutationBatcher.swift:73-294, SHA3BatchHasher.swift:81-264;
// Metal kernels HashMerkleKernels.metal:428-478, 758-909).
//
// One permutation per thread, state in registers.  Contiguous 200-byte states are
// staged through shared memory with 16-byte coalesced loads; other strides load
// lane by lane.
#include "azk_internal.h"
#include "azk_message.cuh"

namespace azk {

// Contiguous states (stride 200, 16-byte aligned base): the CTA copies its
// blockDim.x states to shared memory with uint4 loads, each thread permutes one.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) keccak_permute_staged(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t count) {
  extern __shared__ uint4 smem4[];
  uint64_t first = (uint64_t)blockIdx.x * THREADS;
  uint32_t n = (uint32_t)((count - first) < (uint64_t)THREADS ? (count - first) : (uint64_t)THREADS);
  const uint4* src = reinterpret_cast<const uint4*>(in + first * 200);
  uint32_t vecs = n * 200 / 16;  // n * 12.5: states pair up into whole vectors
  uint32_t tail_bytes = (n * 200) % 16;
  for (uint32_t v = threadIdx.x; v < vecs; v += THREADS) smem4[v] = __ldg(src + v);
  if (tail_bytes && threadIdx.x == 0) {
    const uint64_t* s8 = reinterpret_cast<const uint64_t*>(in + first * 200 + (uint64_t)vecs * 16);
    reinterpret_cast<uint64_t*>(smem4 + vecs)[0] = s8[0];
  }
  __syncthreads();
  if (threadIdx.x < n) {
    uint64_t* st = reinterpret_cast<uint64_t*>(smem4) + threadIdx.x * 25;
    uint64_t a[25];
#pragma unroll
    for (int i = 0; i < 25; i++) a[i] = st[i];
    keccak_f1600(a);
#pragma unroll
    for (int i = 0; i < 25; i++) st[i] = a[i];
  }
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(out + first * 200);
  for (uint32_t v = threadIdx.x; v < vecs; v += THREADS) dst[v] = smem4[v];
  if (tail_bytes && threadIdx.x == 0) {
    uint64_t* d8 = reinterpret_cast<uint64_t*>(out + first * 200 + (uint64_t)vecs * 16);
    d8[0] = reinterpret_cast<uint64_t*>(smem4 + vecs)[0];
  }
}

// Any stride that is a multiple of 8 bytes: lane-by-lane loads and stores; bytes
// of an output stride beyond 200 are zeroed (the reference zeroes its output
// buffer when outputStride > 200, KeccakF1600PermutationBatcher.swift:161-164).
__global__ void __launch_bounds__(256) keccak_permute_strided(const uint8_t* __restrict__ in, uint64_t in_stride, uint8_t* __restrict__ out,
                                                              uint64_t out_stride, uint64_t count) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint64_t* s = reinterpret_cast<const uint64_t*>(in + i * in_stride);
  uint64_t a[25];
#pragma unroll
  for (int k = 0; k < 25; k++) a[k] = __ldg(s + k);
  keccak_f1600(a);
  uint64_t* d = reinterpret_cast<uint64_t*>(out + i * out_stride);
#pragma unroll
  for (int k = 0; k < 25; k++) d[k] = a[k];
  for (uint64_t k = 25; k < out_stride / 8; k++) d[k] = 0;
}

cudaError_t launch_keccak_permute(const uint8_t* in, uint64_t in_stride, uint8_t* out, uint64_t out_stride, uint64_t count, uint32_t threads,
                                  cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  bool staged = in_stride == 200 && out_stride == 200 && ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0);
  if (staged) {
    constexpr int T = 128;
    uint64_t blocks = (count + T - 1) / T;
    keccak_permute_staged<T><<<(unsigned)blocks, T, T * 200, s>>>(in, out, count);
  } else {
    uint32_t t = threads ? threads : 256;
    if (t > 256) t = 256;
    keccak_permute_strided<<<(unsigned)((count + t - 1) / t), t, 0, s>>>(in, in_stride, out, out_stride, count);
  }
  return cudaGetLastError();
}

// A digest and the zeroed padding up to out_stride.
__device__ __forceinline__ void store_digest(uint8_t* o, uint64_t out_stride, const uint64_t (&d)[4], uint32_t out_align) {
  if (out_align >= 8) {
    uint64_t* o8 = reinterpret_cast<uint64_t*>(o);
    if (out_align >= 16) {
      reinterpret_cast<ulonglong2*>(o8)[0] = make_ulonglong2(d[0], d[1]);
      reinterpret_cast<ulonglong2*>(o8)[1] = make_ulonglong2(d[2], d[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) o8[k] = d[k];
    }
    for (uint64_t k = 4; k < out_stride / 8; k++) o8[k] = 0;
  } else {
#pragma unroll
    for (int k = 0; k < 32; k++) o[k] = (uint8_t)(d[k >> 3] >> (8 * (k & 7)));
    for (uint64_t k = 32; k < out_stride; k++) o[k] = 0;
  }
}

// A message into 4-byte units, at its own offset within the first, by this warp (CTAs are
// whole warps); its loads are all in flight at once.
static constexpr uint32_t kEdgeUnits = 35;  // 3 + 136 bytes
__device__ __forceinline__ const uint8_t* copy_message(uint32_t* units, const uint8_t* p, uint32_t len) {
  uint8_t* const to = reinterpret_cast<uint8_t*>(units) + (reinterpret_cast<uintptr_t>(p) & 3);
  const uint32_t lane = threadIdx.x & 31;
  uint8_t b[5];
#pragma unroll
  for (uint32_t j = 0; j < 5; j++) b[j] = lane + 32 * j < len ? __ldg(p + lane + 32 * j) : 0;
#pragma unroll
  for (uint32_t j = 0; j < 5; j++)
    if (lane + 32 * j < len) to[lane + 32 * j] = b[j];
  return to;
}

// One message per thread.  LEN: the length where it is compiled in (0: `len`).
// Messages that are not 8-byte aligned are read in whole 4-byte units, which for the
// batch's first and last message may reach outside the caller's buffer: the warps that
// hold these copy them to shared memory, byte by byte, and read them there.  (Host call
// included, without the copy / so / with a second, byte-exact reader in the same code: 16
// messages of 100 bytes at stride 103 29.0, 29.3, 32.9 us; 2^20 of 99 bytes 282, 280, 279.
// Byte loads throughout: 354 us at 256 threads per CTA, 287 in units.)
template <uint32_t LEN>
__global__ void __launch_bounds__(256) hash_batch(const uint8_t* __restrict__ in, uint64_t stride, uint32_t len, uint32_t suffix,
                                                  uint8_t* __restrict__ out, uint64_t out_stride, uint64_t count, uint32_t aligned8, uint32_t out_align) {
  __shared__ uint32_t s_edge[2][kEdgeUnits];
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n = LEN ? LEN : len;
  const uint8_t* p = in + i * stride;
  if (!aligned8) {
    const uint64_t w = i - (threadIdx.x & 31);  // the warp's first message
    const uint8_t *first = nullptr, *last = nullptr;
    if (w == 0) first = copy_message(s_edge[0], in, n);
    if (w < count && count - 1 - w < 32) last = copy_message(s_edge[1], in + (count - 1) * stride, n);
    __syncwarp();
    if (i + 1 == count && last) p = last;
    if (i == 0 && first) p = first;
  }
  if (i >= count) return;
  uint64_t d[4];
  hash_message<false, AnyLoads, ReadOnlyLoads>(p, n, suffix, aligned8 != 0, d);
  store_digest(out + i * out_stride, out_stride, d, out_align);
}

// Threads per CTA when the plan leaves the choice: the SMs' shares of the messages
// differ by at most one CTA, and a CTA's registers are given back only when its last
// warp ends, so small CTAs (2^20 messages of 99 bytes: 256 threads 287 us, 64 and 128
// 267; 2^22 of 64 bytes 1006, 991 and 991; 30,000 of 55 bytes 17.0, 17.5 and 16.8).
cudaError_t launch_hash_batch(const uint8_t* in, uint64_t stride, uint32_t len, uint32_t suffix, uint8_t* out, uint64_t out_stride, uint64_t count,
                              uint32_t threads, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  uint32_t t = threads ? threads : 128;
  if (t > 256) t = 256;
  const unsigned blocks = (unsigned)((count + t - 1) / t);
  const uint32_t aligned8 = (((uintptr_t)in & 7) == 0 && (stride & 7) == 0) ? 1 : 0;
  const uintptr_t o = (uintptr_t)out | (uintptr_t)out_stride;
  const uint32_t out_align = (o & 15) == 0 ? 16 : (o & 7) == 0 ? 8 : 1;
  switch (len) {
    case 32: hash_batch<32><<<blocks, t, 0, s>>>(in, stride, len, suffix, out, out_stride, count, aligned8, out_align); break;
    case 64: hash_batch<64><<<blocks, t, 0, s>>>(in, stride, len, suffix, out, out_stride, count, aligned8, out_align); break;
    case 128: hash_batch<128><<<blocks, t, 0, s>>>(in, stride, len, suffix, out, out_stride, count, aligned8, out_align); break;
    case 136: hash_batch<136><<<blocks, t, 0, s>>>(in, stride, len, suffix, out, out_stride, count, aligned8, out_align); break;
    default: hash_batch<0><<<blocks, t, 0, s>>>(in, stride, len, suffix, out, out_stride, count, aligned8, out_align); break;
  }
  return cudaGetLastError();
}

}  // namespace azk

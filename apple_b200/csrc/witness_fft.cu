// Monomial -> Chebyshev coefficients by fast convolution, for long witness columns
// (witness_kernels.cu has the direct sum, whose work grows with the square of the
// column).  With x = (z + 1/z) / 2, P(x) = sum_m c_m T_m(x) is the Laurent
// polynomial sum_m l_m z^m, c_0 = l_0, c_m = 2 l_m, and (x - 1) / (x + 1) is the
// square of (z - 1) / (z + 1).  So with n = 2^k coefficients, D = n - 1:
//   1. P(y - 1)                       = sum_i b_i y^i                  (shift)
//   2. sum_j b_(D-j) 2^(D-j) u^j at u = 1 - w: coefficients q_i of w^i (shift)
//      -- now P(x) (1 - w)^D = Q(w) for x = (1 + w) / (1 - w)
//   3. R(v) = Q(v^2), shifted by one: coefficients r_i of degree i <= D (the even
//      and the odd ones are two products with the n values of q)
//   4. the upper half of sum_i r_i (-2)^i y^(2D-i) at y = z + 1 (shift), whose
//      coefficient of z^(D+m) is 4^D l_m.
// A Taylor shift by s is G_i = sum_(k>=i) F_k s^(k-i) / (k-i)! with F_k = f_k k!
// and g_i = G_i / i!: a correlation with a fixed M31 sequence, done as a cyclic one
// of size 2n by number-theoretic transforms over CM31 = M31[i], whose elements of
// norm one (the circle group) have order 2^31.  The fixed sequences are M31, so one
// CM31 transform carries two M31 columns: a QM31 column is two CM31 sequences, and
// two lifted M31 columns are one.  All arithmetic is exact.
//
// A transform of 2^lm values is natural order in, bit-reversed out, block b of a
// stage multiplied by the root Z[b] = w^bitrev(b) (the same table prefix for every
// stage and size); the inverse runs the stages backwards on bit-reversed input.
// Stages above bit 12 (10) run on strided tiles of 4096 (1024) values, the low ones
// on contiguous tiles: there the forward stages, the product with the fixed
// sequence's transform and the inverse stages are one kernel, so a convolution is
// three passes over memory.  What bounds them is integer issue: about
// 52 instructions per QM31 butterfly.  Two columns of 2^19 QM31 (lifted M31)
// coefficients: 0.83 (0.34) ms, against 175.9 ms for the direct sum's O(n^2).
#include "azk_field.cuh"
#include "azk_internal.h"

namespace azk {
namespace {

// Values of a tile: 4096 for large transforms, 1024 (and strided stages from bit 10
// up) for those of at most 2^kShortLog values, which would leave most SMs without a
// tile and whose time is the latency of one tile (columns of 2^17: 325 us with long
// tiles, 255 with short ones; of 2^14: 246 and 116; of 2^18 495 and no strided tile
// with 64-byte rows).
constexpr uint32_t kLongTile = 12, kShortTile = 10, kShortLog = 18;
// Threads of a tile's CTA.  A long tile's stages are chains of shared-memory round
// trips in few CTAs (13 of 64 warps resident at 256 threads): lifted columns of 2^21
// 1032 us with 256, 968 with 512, 972 with 1024; of 2^18 234, 196 and 186; QM31 ones of 2^21
// 3241, 3072 and 3544.  A short tile has work for 256.
template <uint32_t TL>
constexpr int kConvThreads = TL >= 12 ? 512 : 256;

// W limbs per value: 2 (one CM31) or 4 (two).
template <int W>
struct Val {
  uint32_t v[W];
};
template <int W>
__device__ __forceinline__ Val<W> ldv(const void* p, uint64_t i) {
  Val<W> r;
  if constexpr (W == 4) {
    const uint4 u = reinterpret_cast<const uint4*>(p)[i];
    r.v[0] = u.x, r.v[1] = u.y, r.v[2] = u.z, r.v[3] = u.w;
  } else {
    const uint2 u = reinterpret_cast<const uint2*>(p)[i];
    r.v[0] = u.x, r.v[1] = u.y;
  }
  return r;
}
template <int W>
__device__ __forceinline__ void stv(void* p, uint64_t i, const Val<W>& r) {
  if constexpr (W == 4)
    reinterpret_cast<uint4*>(p)[i] = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else
    reinterpret_cast<uint2*>(p)[i] = make_uint2(r.v[0], r.v[1]);
}
// a b + c d for values <= p, reduced to at most p: the sum is below 2^63, so its
// three 31-bit parts add up to at most 2p.
__device__ __forceinline__ uint32_t mul2_add(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  const uint64_t v = (uint64_t)a * b + (uint64_t)c * d;
  const uint32_t hi = (uint32_t)(v >> 31);
  return m31_reduce_once(((uint32_t)v & kP) + (hi & kP) + (hi >> 31));
}
template <int W>
__device__ __forceinline__ Val<W> cmul(const Val<W>& x, uint2 t) {
  Val<W> r;
  const uint32_t nt = kP - t.y;
#pragma unroll
  for (int k = 0; k < W; k += 2) {
    r.v[k] = mul2_add(x.v[k], t.x, x.v[k + 1], nt);
    r.v[k + 1] = mul2_add(x.v[k], t.y, x.v[k + 1], t.x);
  }
  return r;
}
template <int W>
__device__ __forceinline__ Val<W> vadd(const Val<W>& a, const Val<W>& b) {
  Val<W> r;
#pragma unroll
  for (int k = 0; k < W; k++) r.v[k] = m31_add(a.v[k], b.v[k]);
  return r;
}
template <int W>
__device__ __forceinline__ Val<W> vsub(const Val<W>& a, const Val<W>& b) {
  Val<W> r;
#pragma unroll
  for (int k = 0; k < W; k++) r.v[k] = m31_sub(a.v[k], b.v[k]);
  return r;
}
template <int W>
__device__ __forceinline__ Val<W> vscale(const Val<W>& a, uint32_t s) {
  Val<W> r;
#pragma unroll
  for (int k = 0; k < W; k++) r.v[k] = m31_mul(a.v[k], s);
  return r;
}
// (l, r) -> (l + r t, l - r t) and its inverse (up to a factor 2).
template <int W>
__device__ __forceinline__ void bfly(Val<W>& l, Val<W>& r, uint2 t) {
  const Val<W> x = cmul(r, t);
  r = vsub(l, x);
  l = vadd(l, x);
}
template <int W>
__device__ __forceinline__ void bfly_inv(Val<W>& l, Val<W>& r, uint2 t) {
  const Val<W> d = vsub(l, r);
  l = vadd(l, r);
  r = cmul(d, make_uint2(t.x, kP - t.y));  // the inverse of a norm-one value is its conjugate
}

// Tile index to shared slot: 16-byte (8-byte) slots whose low three bits are XORed
// with bits 3 and 4, so that the strided accesses of every stage pair on bits
// (p, p - 1), p odd (and p = 4), fall on distinct banks.
__device__ __forceinline__ uint32_t slot(uint32_t i) { return i ^ ((i >> 3) & 1u) ^ (((i >> 4) & 1u) * 6u); }

// Stages on the m row bits of a tile of 2^(m + c) values (local index (row << c) |
// col), two per shared-memory round trip.  Row bit j's block is (hi << (m-1-j)) +
// (row >> (j+1)).  Starts and ends with the tile in shared memory and every thread
// past a barrier.  top: row bits >= top are already done (forward) or not wanted.
template <int W, int THREADS>
__device__ __forceinline__ void forward_stages(Val<W>* sm, uint32_t m, uint32_t top, uint32_t c, uint64_t hi, const uint2* __restrict__ roots) {
  const uint32_t T = 1u << (m + c);
  int j = (int)top - 1;
  for (; j >= 1; j -= 2) {
    const uint32_t p = (uint32_t)j + c;  // stages on local bits p and p - 1
    const uint32_t low = (1u << (p - 1)) - 1;
    for (uint32_t k = threadIdx.x; k < T / 4; k += THREADS) {
      const uint32_t e = ((k & ~low) << 2) | (k & low);
      const uint64_t b = (hi << (m - 1 - j)) + (e >> (c + j + 1));
      const uint2 t1 = __ldg(roots + b);
      const uint4 t2 = __ldg(reinterpret_cast<const uint4*>(roots) + b);  // entries 2b, 2b + 1
      const uint32_t s0 = slot(e), s1 = slot(e | (1u << (p - 1))), s2 = slot(e | (1u << p)), s3 = slot(e | (3u << (p - 1)));
      Val<W> v0 = sm[s0], v1 = sm[s1], v2 = sm[s2], v3 = sm[s3];
      bfly(v0, v2, t1);
      bfly(v1, v3, t1);
      bfly(v0, v1, make_uint2(t2.x, t2.y));
      bfly(v2, v3, make_uint2(t2.z, t2.w));
      sm[s0] = v0, sm[s1] = v1, sm[s2] = v2, sm[s3] = v3;
    }
    __syncthreads();
  }
  if (j == 0) {
    for (uint32_t k = threadIdx.x; k < T / 2; k += THREADS) {
      const uint32_t low = (1u << c) - 1, e = ((k & ~low) << 1) | (k & low);
      const uint2 t = __ldg(roots + (hi << (m - 1)) + (e >> (c + 1)));
      const uint32_t s0 = slot(e), s1 = slot(e | (1u << c));
      Val<W> l = sm[s0], r = sm[s1];
      bfly(l, r, t);
      sm[s0] = l, sm[s1] = r;
    }
    __syncthreads();
  }
}
template <int W, int THREADS>
__device__ __forceinline__ void inverse_stages(Val<W>* sm, uint32_t m, uint32_t c, uint64_t hi, const uint2* __restrict__ roots) {
  const uint32_t T = 1u << (m + c);
  uint32_t j = 0;
  if (m & 1) {
    for (uint32_t k = threadIdx.x; k < T / 2; k += THREADS) {
      const uint32_t low = (1u << c) - 1, e = ((k & ~low) << 1) | (k & low);
      const uint2 t = __ldg(roots + (hi << (m - 1)) + (e >> (c + 1)));
      const uint32_t s0 = slot(e), s1 = slot(e | (1u << c));
      Val<W> l = sm[s0], r = sm[s1];
      bfly_inv(l, r, t);
      sm[s0] = l, sm[s1] = r;
    }
    __syncthreads();
    j = 1;
  }
  for (; j + 1 < m + 0u; j += 2) {
    const uint32_t p = j + 1 + c;  // stages on local bits p - 1, then p
    const uint32_t low = (1u << (p - 1)) - 1;
    for (uint32_t k = threadIdx.x; k < T / 4; k += THREADS) {
      const uint32_t e = ((k & ~low) << 2) | (k & low);
      const uint64_t b = (hi << (m - 2 - j)) + (e >> (c + j + 2));
      const uint2 t1 = __ldg(roots + b);
      const uint4 t2 = __ldg(reinterpret_cast<const uint4*>(roots) + b);
      const uint32_t s0 = slot(e), s1 = slot(e | (1u << (p - 1))), s2 = slot(e | (1u << p)), s3 = slot(e | (3u << (p - 1)));
      Val<W> v0 = sm[s0], v1 = sm[s1], v2 = sm[s2], v3 = sm[s3];
      bfly_inv(v0, v1, make_uint2(t2.x, t2.y));
      bfly_inv(v2, v3, make_uint2(t2.z, t2.w));
      bfly_inv(v0, v2, t1);
      bfly_inv(v1, v3, t1);
      sm[s0] = v0, sm[s1] = v1, sm[s2] = v2, sm[s3] = v3;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ uint32_t pow2_m31(uint64_t e) { return 1u << (e % 31); }
// 2^-e mod p
__device__ __forceinline__ uint32_t pow2_inv_m31(uint64_t e) { return 1u << ((31 - e % 31) % 31); }

// Input i (< n) of convolution `step`: the previous one's raw output (a factor
// 2^lm too large, which the power of two takes out) in the order and with the
// factors of the text above.
enum Step { kShift1 = 0, kShift2 = 1, kParity = 2, kShift4 = 3, kTable = 4 };
template <int W, int STEP>
__device__ __forceinline__ Val<W> conv_input(const WitnessConv& a, uint32_t column, uint64_t i) {
  const uint64_t n = 1ull << (a.lm - 1), D = n - 1;
  Val<W> r;
  if constexpr (STEP == kTable) {
    // the fixed sequence s_j (0 <= j < n) at position -j: 1/j!, 1/(2j)! or 1/(2j-1)!
    const uint32_t e = a.table == 0 ? a.ifact[i] : a.table == 1 ? a.ifact[2 * i] : i ? a.ifact[2 * i - 1] : 0u;
#pragma unroll
    for (int k = 0; k < W; k++) r.v[k] = 0;
    r.v[0] = e;
    return r;
  } else if constexpr (STEP == kShift1) {
    const uint32_t f = a.fact[i];
    if constexpr (W == 2) {
      r.v[0] = i < a.count_x ? m31_mul(a.x[i].x, f) : 0u;
      r.v[1] = i < a.count_y ? m31_mul(a.y[i].x, f) : 0u;
      return r;
    } else {
      const uint4* col = column ? a.y : a.x;
      if (i < (column ? a.count_y : a.count_x)) return vscale(ldv<W>(col, i), f);
#pragma unroll
      for (int k = 0; k < W; k++) r.v[k] = 0;
      return r;
    }
  } else if constexpr (STEP == kShift2) {
    const uint64_t k = D - i;
    const uint32_t w = m31_mul(m31_mul(a.ifact[k], a.fact[i]), pow2_m31(k + 31 - a.lm % 31));
    return vscale(ldv<W>(a.c + column * a.c_stride, k), w);
  } else if constexpr (STEP == kParity) {
    uint32_t w = m31_mul(m31_mul(a.ifact[i], a.fact[2 * i]), pow2_inv_m31(a.lm));
    if (i & 1) w = m31_neg(w);
    return vscale(ldv<W>(a.c + column * a.c_stride, i), w);
  } else {
    const uint64_t k = D - i;  // r_k (-2)^k at y^(D + i), r_k = G_k / k!
    uint32_t w = m31_mul(m31_mul(a.ifact[k], a.fact[D + i]), pow2_m31(k + 31 - a.lm % 31));
    if (k & 1) w = m31_neg(w);
    return vscale(ldv<W>(a.c + (k & 1 ? a.odd : 0) + column * (a.c_stride / 2), k >> 1), w);
  }
}

// The strided pass of the forward transform (stages above bit 12): inputs from
// conv_input (zero from n on, so the first stage only copies), all 2n values to `t`.
template <int W, int STEP, uint32_t TL>
__global__ void __launch_bounds__(kConvThreads<TL>) conv_high_kernel(const WitnessConv a) {
  constexpr uint32_t kTile = 1u << TL;
  constexpr int kThreads = kConvThreads<TL>;
  dependent_begin();
  extern __shared__ __align__(16) uint8_t smem[];
  Val<W>* sm = reinterpret_cast<Val<W>*>(smem);
  const uint32_t m = a.lm - TL, c = TL - m;
  const uint64_t col0 = (uint64_t)blockIdx.x << c;
  const uint64_t M = 1ull << a.lm, n = M / 2;
  for (uint32_t L = threadIdx.x; L < kTile / 2; L += kThreads) {
    const uint64_t i = ((uint64_t)(L >> c) << TL) | col0 | (L & ((1u << c) - 1));
    Val<W> v;
    if constexpr (STEP == kTable) {
      // positions M - j: the upper half, and position 0
      const Val<W> z = conv_input<W, STEP>(a, 0, i == 0 ? 0 : n - i);
      Val<W> lo = z;
      if (i != 0) {
#pragma unroll
        for (int k = 0; k < W; k++) lo.v[k] = 0;
      }
      v = z;
      if (i == 0) {
#pragma unroll
        for (int k = 0; k < W; k++) v.v[k] = 0;
      }
      // first stage: root 1
      sm[slot(L)] = vadd(lo, v);
      sm[slot(L + kTile / 2)] = vsub(lo, v);
    } else {
      v = conv_input<W, STEP>(a, blockIdx.y, i);
      sm[slot(L)] = v;
      sm[slot(L + kTile / 2)] = v;
    }
  }
  __syncthreads();
  forward_stages<W, kThreads>(sm, m, m - 1, c, 0, a.roots);
  uint8_t* t = static_cast<uint8_t*>(a.t) + blockIdx.y * a.t_stride;
  for (uint32_t L = threadIdx.x; L < kTile; L += kThreads)
    stv<W>(t, ((uint64_t)(L >> c) << TL) | col0 | (L & ((1u << c) - 1)), sm[slot(L)]);
}

// The low stages on contiguous tiles: forward, times the fixed sequence's transform
// (blockIdx.z picks one of two), inverse, from `t` to u[z].
template <int W, uint32_t TL>
__global__ void __launch_bounds__(kConvThreads<TL>) conv_low_kernel(const WitnessConv a) {
  constexpr uint32_t kTile = 1u << TL;
  constexpr int kThreads = kConvThreads<TL>;
  dependent_begin();
  extern __shared__ __align__(16) uint8_t smem[];
  Val<W>* sm = reinterpret_cast<Val<W>*>(smem);
  const uint64_t base = (uint64_t)blockIdx.x << TL;
  const uint8_t* t = static_cast<const uint8_t*>(a.t) + blockIdx.y * a.t_stride;
  for (uint32_t L = threadIdx.x; L < kTile; L += kThreads) sm[slot(L)] = ldv<W>(t, base + L);
  __syncthreads();
  forward_stages<W, kThreads>(sm, TL, TL, 0, blockIdx.x, a.roots);
  if (a.k[0] == nullptr) {  // a fixed sequence's own transform
    for (uint32_t L = threadIdx.x; L < kTile; L += kThreads) {
      const Val<W> v = sm[slot(L)];
      static_cast<uint2*>(a.u[0])[base + L] = make_uint2(v.v[0], v.v[1]);
    }
    return;
  }
  const uint2* kf = a.k[blockIdx.z];
  for (uint32_t L = threadIdx.x; L < kTile; L += kThreads) {
    const uint32_t s = slot(L);
    sm[s] = cmul(sm[s], __ldg(kf + ((base + L) ^ a.flip)));
  }
  __syncthreads();
  inverse_stages<W, kThreads>(sm, TL, 0, blockIdx.x, a.roots);
  uint8_t* u = static_cast<uint8_t*>(a.u[blockIdx.z]) + blockIdx.y * a.t_stride;
  for (uint32_t L = threadIdx.x; L < kTile; L += kThreads) stv<W>(u, base + L, sm[slot(L)]);
}

// The strided inverse pass; the wanted outputs to o[z].
template <int W, uint32_t TL>
__global__ void __launch_bounds__(kConvThreads<TL>) conv_out_kernel(const WitnessConv a) {
  constexpr uint32_t kTile = 1u << TL;
  constexpr int kThreads = kConvThreads<TL>;
  dependent_begin();
  extern __shared__ __align__(16) uint8_t smem[];
  Val<W>* sm = reinterpret_cast<Val<W>*>(smem);
  const uint32_t m = a.lm - TL, c = TL - m;
  const uint64_t col0 = (uint64_t)blockIdx.x << c;
  const uint8_t* u = static_cast<const uint8_t*>(a.u[blockIdx.z]) + blockIdx.y * a.t_stride;
  for (uint32_t L = threadIdx.x; L < kTile; L += kThreads)
    sm[slot(L)] = ldv<W>(u, ((uint64_t)(L >> c) << TL) | col0 | (L & ((1u << c) - 1)));
  __syncthreads();
  inverse_stages<W, kThreads>(sm, m, c, 0, a.roots);
  uint8_t* o = a.o[blockIdx.z] + blockIdx.y * a.o_stride;
  for (uint32_t L = threadIdx.x; L < kTile / 2; L += kThreads) {
    const uint64_t i = ((uint64_t)(L >> c) << TL) | col0 | (L & ((1u << c) - 1));
    if (i < a.outputs) stv<W>(o, i, sm[slot(L)]);
  }
}

// Root table: Z[b] = w^bitrev(b), w of order 2^(log + 1), b < 2^log.
__global__ void roots_kernel(uint2* __restrict__ roots, uint32_t log) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >> log) return;
  const cpoint p = cp_from_index(bit_reverse(b, log) << (30 - log));
  roots[b] = make_uint2(p.x, p.y);
}

// c_m = (m ? 2 : 1) l_m from the last convolution, in place, then the levels of the
// Chebyshev -> line-basis recursion (witness_kernels.cu) down to blocks of w = 2^lw
// values, up to four per launch: the elements {b w + r, b w + w - r} of a block of
// 2^k w values only meet one another on those levels, so a thread takes one r.
// Levels run from blocks of `s` = w << k values to blocks of w values.
constexpr int kLineK = 3;
template <int W>
__device__ __forceinline__ Val<W> cheb_value(const WitnessConv& a, const uint8_t* c, uint64_t i, bool first) {
  Val<W> v = ldv<W>(c, i);
  if (first) {
    const uint64_t D = (1ull << (a.lm - 1)) - 1, m = i;
    // 2^-lm 4^-D, doubled for m > 0
    const uint32_t w = m31_mul(a.ifact[D + m], pow2_inv_m31((uint64_t)a.lm + 2 * D - (m ? 1 : 0)));
    v = vscale(v, w);
  }
  return v;
}
template <int W>
__global__ void __launch_bounds__(256) line_levels_kernel(const WitnessConv a, uint32_t lw, uint32_t k, uint32_t first) {
  dependent_begin();
  uint8_t* c = a.c + blockIdx.y * a.c_stride;
  const uint64_t w = 1ull << lw, n = 1ull << (a.lm - 1);
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t per = w / 2 + 1;  // r = 0 .. w / 2
  if (g >= (n >> (lw + k)) * per) return;
  const uint64_t blk = g / per, r = g % per, base = blk << (lw + k);
  const uint32_t nb = 1u << k;
  Val<W> lo[1 << kLineK], hi[1 << kLineK];  // b w + r, b w + w - r
#pragma unroll
  for (int b = 0; b < (1 << kLineK); b++) {
    if (b >= (int)nb) continue;
    lo[b] = cheb_value<W>(a, c, base + b * w + r, first != 0);
    if (r != 0 && 2 * r != w) hi[b] = cheb_value<W>(a, c, base + b * w + w - r, first != 0);
  }
  // level of blocks of 2^l w values: lo[b] (offset b w + r) meets hi[b'] with
  // b + b' = 2^l - 1, and hi[b] meets lo[b'] likewise; r = 0 meets r = 0 (b + b' = 2^l)
#pragma unroll
  for (int l = kLineK; l >= 0; l--) {
    if (l > (int)k) continue;
#pragma unroll
    for (int q = 0; q < (1 << kLineK); q += (1 << l)) {
      if (q >= (int)nb) continue;
      if (r == 0) {
#pragma unroll
        for (int b = 1; 2 * b < (1 << l); b++) {
          const Val<W> x = lo[q + b], y = lo[q + (1 << l) - b];
          lo[q + b] = vsub(x, y);
          lo[q + (1 << l) - b] = vadd(y, y);
        }
      } else if (2 * r == w) {
        // offset (b + 1/2) w meets offset (2^l - b - 1/2) w
#pragma unroll
        for (int b = 0; 2 * b + 1 < (1 << l); b++) {
          const Val<W> x = lo[q + b], y = lo[q + (1 << l) - 1 - b];
          lo[q + b] = vsub(x, y);
          lo[q + (1 << l) - 1 - b] = vadd(y, y);
        }
      } else {
#pragma unroll
        for (int b = 0; b < (1 << l); b++) {
          const int o = (1 << l) - 1 - b;
          // the pair (lo[b], hi[o]): the smaller offset is the low one
          if (2 * b < (1 << l) && (b < o || l == 0)) {
            Val<W> x = lo[q + b], y = hi[q + o];
            lo[q + b] = vsub(x, y);
            hi[q + o] = vadd(y, y);
            if (l > 0) {
              x = hi[q + b], y = lo[q + o];
              hi[q + b] = vsub(x, y);
              lo[q + o] = vadd(y, y);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int b = 0; b < (1 << kLineK); b++) {
    if (b >= (int)nb) continue;
    stv<W>(c, base + b * w + r, lo[b]);
    if (r != 0 && 2 * r != w) stv<W>(c, base + b * w + w - r, hi[b]);
  }
}

// The levels of blocks of at most 2^lt values, in shared memory, and the
// interleaved output out[2i] = x, out[2i + 1] = y; zeros from n to the capacity.
template <int W>
__global__ void __launch_bounds__(512) line_out_kernel(const WitnessConv a, uint32_t lt, uint32_t first, uint4* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem[];
  dependent_begin();
  const uint64_t n = 1ull << (a.lm - 1);
  const uint32_t T = 1u << lt;
  const uint64_t base = (uint64_t)blockIdx.x << lt;
  if (base >= n) {
    for (uint32_t i = threadIdx.x; i < 2 * T; i += blockDim.x) out[2 * base + i] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  constexpr int kCols = W == 4 ? 2 : 1;
  Val<W>* sm = reinterpret_cast<Val<W>*>(smem);
#pragma unroll
  for (int col = 0; col < kCols; col++)
    for (uint32_t i = threadIdx.x; i < T; i += blockDim.x) sm[col * T + i] = cheb_value<W>(a, a.c + col * a.c_stride, base + i, first != 0);
  __syncthreads();
  for (uint32_t ls = lt; ls >= 2; ls--) {
    const uint32_t half = 1u << (ls - 1), mask = half - 1;
    for (uint32_t g = threadIdx.x; g < T / 2; g += blockDim.x) {
      const uint32_t i = g & mask, b = (g >> (ls - 1)) << ls;
      if (i == 0) continue;
#pragma unroll
      for (int col = 0; col < kCols; col++) {
        Val<W>*x = sm + col * T + b + i, *y = sm + col * T + b + 2 * half - i;
        const Val<W> l = *x, h = *y;
        *x = vsub(l, h);
        *y = vadd(h, h);
      }
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < T; i += blockDim.x) {
    if constexpr (W == 4) {
      stv<W>(out, 2 * (base + i), sm[i]);
      stv<W>(out, 2 * (base + i) + 1, sm[T + i]);
    } else {
      out[2 * (base + i)] = make_uint4(sm[i].v[0], 0u, 0u, 0u);
      out[2 * (base + i) + 1] = make_uint4(sm[i].v[1], 0u, 0u, 0u);
    }
  }
}

// A convolution from conv_input (HIGH) or from the values that one left in `t`: `outs`
// products at once.
template <int W, int STEP, uint32_t TL, bool HIGH>
cudaError_t run_conv_tiles(const WitnessConv& a, uint32_t columns, uint32_t outs, cudaStream_t s) {
  const uint32_t tiles = 1u << (a.lm - TL);
  const size_t smem = (size_t)4 * W << TL;
  cudaError_t e = cudaSuccess;
  if constexpr (HIGH) e = launch_dependent(conv_high_kernel<W, STEP, TL>, dim3(tiles, columns), dim3(kConvThreads<TL>), smem, s, a);
  if (e == cudaSuccess) e = launch_dependent(conv_low_kernel<W, TL>, dim3(tiles, columns, outs), dim3(kConvThreads<TL>), smem, s, a);
  if (e == cudaSuccess && STEP != kTable) e = launch_dependent(conv_out_kernel<W, TL>, dim3(tiles, columns, outs), dim3(kConvThreads<TL>), smem, s, a);
  return e;
}
template <int W, int STEP, bool HIGH = true>
cudaError_t run_conv(const WitnessConv& a, uint32_t columns, uint32_t outs, cudaStream_t s) {
  return a.lm <= kShortLog ? run_conv_tiles<W, STEP, kShortTile, HIGH>(a, columns, outs, s) : run_conv_tiles<W, STEP, kLongTile, HIGH>(a, columns, outs, s);
}

constexpr uint32_t kLineTileLog = 11;  // 2 columns x 2048 x 16 bytes of shared memory
constexpr uint32_t kLineTileShort = 9;  // up to 2^(kShortLog - 1) values: more tiles, shorter ones

// Line basis of the two columns in a.c (n values each; first: still raw convolution
// outputs): blocks of n, n / 2, ... values, four levels a launch, then the shared tile.
template <int W>
cudaError_t line_basis(const WitnessConv& a, uint32_t first, uint4* out, uint64_t capacity, cudaStream_t s) {
  const uint32_t columns = W == 4 ? 2 : 1;
  const uint64_t n = 1ull << (a.lm - 1);
  const uint32_t ln = a.lm - 1, tile = a.lm <= kShortLog ? kLineTileShort : kLineTileLog, lt = ln < tile ? ln : tile;
  for (uint32_t ls = ln; ls > lt;) {
    const uint32_t k = ls - lt - 1 < (uint32_t)kLineK ? ls - lt - 1 : kLineK, lw = ls - k;
    const uint64_t threads = (n >> ls) * ((1ull << lw) / 2 + 1);
    const cudaError_t e = launch_dependent(line_levels_kernel<W>, dim3((unsigned)((threads + 255) / 256), columns), dim3(256), 0, s, a, lw, k, first);
    if (e != cudaSuccess) return e;
    first = 0;
    ls = lw - 1;
  }
  return launch_dependent(line_out_kernel<W>, dim3((unsigned)(capacity >> lt)), dim3(512), (size_t)columns * 4 * W << lt, s, a, lt, first, out);
}

template <int W>
cudaError_t transform(WitnessConv a, const WitnessKernels& kr, uint4* out, uint64_t capacity, cudaStream_t s) {
  const uint32_t columns = W == 4 ? 2 : 1;
  const uint64_t n = 1ull << (a.lm - 1);
  // a single-output convolution's low stages run in place
  void* const u[2] = {a.u[0], a.u[1]};
  a.u[0] = a.t;
  a.o[0] = a.c;
  a.o_stride = a.c_stride;
  a.outputs = n;
  // 1: shift by -1: the sequence (-1)^j / j!, whose transform is that of 1 / j! half
  // a turn on (the lowest bit of a bit-reversed index)
  a.k[0] = kr.k[0];
  a.flip = 1;
  cudaError_t e = run_conv<W, kShift1>(a, columns, 1, s);
  if (e != cudaSuccess) return e;
  a.flip = 0;
  if ((e = run_conv<W, kShift2>(a, columns, 1, s)) != cudaSuccess) return e;
  // the even and the odd values take the place of c, which only the first pass reads
  a.k[0] = kr.k[1], a.k[1] = kr.k[2];
  a.u[0] = u[0], a.u[1] = u[1];
  a.odd = columns * a.c_stride / 2;
  a.o[0] = a.c, a.o[1] = a.c + a.odd;
  a.o_stride = a.c_stride / 2;
  a.outputs = n / 2;
  if ((e = run_conv<W, kParity>(a, columns, a.u[1] ? 2 : 1, s)) != cudaSuccess) return e;
  if (!a.u[1]) {
    a.k[0] = kr.k[2];
    a.u[0] = a.t;
    a.o[0] = a.o[1];
    if ((e = run_conv<W, kParity, false>(a, columns, 1, s)) != cudaSuccess) return e;
  }
  a.k[0] = kr.k[0];
  a.u[0] = a.t;
  a.o[0] = a.c;
  a.o_stride = a.c_stride;
  a.outputs = n;
  if ((e = run_conv<W, kShift4>(a, columns, 1, s)) != cudaSuccess) return e;
  return line_basis<W>(a, 1, out, capacity, s);
}

template <class K>
cudaError_t opt_in(K k, size_t bytes) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

cudaError_t launch_witness_roots(uint2* roots, uint32_t log, cudaStream_t s) {
  roots_kernel<<<((1u << log) + 255) / 256, 256, 0, s>>>(roots, log);
  return cudaGetLastError();
}

// Transforms of the three fixed sequences for convolutions of 2^a.lm values; `a`
// holds the tables and one column of scratch `t` (2^lm values of 8 bytes).
cudaError_t launch_witness_fft_tables(WitnessConv a, const WitnessKernels& kr, cudaStream_t s) {
  a.k[0] = nullptr;
  for (uint32_t j = 0; j < 3; j++) {
    a.table = j;
    a.u[0] = const_cast<uint2*>(kr.k[j]);
    const cudaError_t e = run_conv<2, kTable>(a, 1, 1, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t prepare_witness_fft() {
  // (the 8-byte forms and the short tiles stay within the default 48 KiB)
  const size_t q = (size_t)16 << kLongTile;
  cudaError_t e = cudaSuccess;
  auto both = [&](cudaError_t r) {
    if (e == cudaSuccess) e = r;
  };
  both(opt_in(conv_high_kernel<4, kShift1, kLongTile>, q)), both(opt_in(conv_high_kernel<4, kShift2, kLongTile>, q));
  both(opt_in(conv_high_kernel<4, kParity, kLongTile>, q)), both(opt_in(conv_high_kernel<4, kShift4, kLongTile>, q));
  both(opt_in(conv_low_kernel<4, kLongTile>, q)), both(opt_in(conv_out_kernel<4, kLongTile>, q));
  both(opt_in(line_out_kernel<4>, (size_t)32 << kLineTileLog));
  return e;
}

cudaError_t launch_witness_fft(const WitnessConv& a, const WitnessKernels& kr, bool lifted, uint4* out, uint64_t capacity, cudaStream_t s) {
  return lifted ? transform<2>(a, kr, out, capacity, s) : transform<4>(a, kr, out, capacity, s);
}

cudaError_t launch_witness_line(const WitnessConv& a, uint4* out, uint64_t capacity, cudaStream_t s) { return line_basis<4>(a, 0, out, capacity, s); }

}  // namespace azk

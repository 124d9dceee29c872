// The sponge transcript on one warp (azk_transcript.cuh has the one-thread form,
// used where many transcripts advance at once): lane m holds state lane m, a frame
// is one message word per lane, and a permutation is WarpKeccak's, so a transcript
// step costs about 2 us instead of the 6 to 7 us of one thread.  Frames and
// squeezing are byte-identical to azk_transcript.cuh.
#pragma once
#include "azk_keccak_coop.cuh"
#include "azk_transcript.cuh"

namespace azk {

// A frame's fixed first bytes: u32 length || domain string || u32 1 || u8 type
// (type zero here), as little-endian words.
struct FrameBase {
  uint64_t w[6];
  uint32_t bytes;
};
constexpr FrameBase frame_base(const char* dom, uint32_t n) {
  FrameBase f{};
  f.bytes = 4 + n + 4 + 1;
  for (uint32_t i = 0; i < f.bytes; i++) {
    uint8_t b = 0;
    if (i < 4) b = (uint8_t)(n >> (8 * i));
    else if (i < 4 + n) b = (uint8_t)dom[i - 4];
    else if (i == 4 + n) b = 1;
    f.w[i / 8] |= (uint64_t)b << (8 * (i % 8));
  }
  return f;
}
struct CircleFrame {
  static constexpr FrameBase base = frame_base("AppleZKProver.CircleFRI.PCS.V1", 30);
};
struct Qm31Frame {
  static constexpr FrameBase base = frame_base("AppleZKProver.QM31FRI.FoldChain", 31);
};
struct SumcheckFrame {
  static constexpr FrameBase base = frame_base("AppleZKProver.M31MultilinearSumcheck", 36);
};

// Word m of the padded one-block message: frame F of type `type` followed by the
// N little-endian u32 words p (a u64 field is two of them), the suffix 0x06 and the
// end padding.  Every position is a compile-time constant, so a lane's word is a
// few selects.
template <class F, int N>
__device__ __forceinline__ uint64_t frame_word(uint32_t m, uint32_t type, const uint32_t (&p)[N]) {
  constexpr FrameBase base = F::base;
  uint64_t v = 0;
#pragma unroll
  for (uint32_t i = 0; i < 6; i++)
    if (m == i) v = base.w[i];
  if (m == (base.bytes - 1) / 8) v |= (uint64_t)type << (8 * ((base.bytes - 1) % 8));
#pragma unroll
  for (uint32_t i = 0; i <= N; i++) {
    const uint32_t x = i < N ? p[i < N ? i : 0] : 0x06u;
    const uint32_t o = base.bytes + 4 * i, w = o / 8, sh = 8 * (o % 8);
    if (m == w) v |= (uint64_t)x << sh;
    if (sh > 32 && m == w + 1) v |= (uint64_t)x >> (64 - sh);
  }
  if (m == 16) v |= kPadEnd;
  return v;
}

// Words squeezed mod p from a state (candidates at or above 2^32 - 2 are skipped):
// the rare rejection is left to the one-thread form.
static __device__ __noinline__ void squeeze_m31_slow(const uint64_t* st, uint32_t count, uint32_t* out) {
  Transcript t;
  for (int i = 0; i < 25; i++) t.st[i] = st[i];
  tr_squeeze_u32(t, count, 2147483647u, out);
}

struct WarpSponge {
  WarpKeccak kf;
  uint32_t lane;
  uint64_t a;

  // `smem`: kWarpKeccakWords words of shared memory of this warp's own.
  __device__ __forceinline__ WarpSponge(uint64_t* smem) : kf(threadIdx.x & 31, smem), lane(threadIdx.x & 31), a(0) {}
  __device__ __forceinline__ void load(const Transcript* t) { a = lane < 25 ? __ldcg(&t->st[lane]) : 0; }
  __device__ __forceinline__ void store(Transcript* t) const {
    if (lane < 25) t->st[lane] = a;
  }
  // One padded block (lane m < 17 passes message word m).
  __device__ __forceinline__ void absorb(uint64_t word) {
    if (lane < 17) a ^= word;
    kf.permute_small(a);
  }
  // Word `lane` of a padded 32-byte message.
  __device__ __forceinline__ uint64_t digest_word(const uint64_t* d) const { return lane < 4 ? d[lane] : lane == 4 ? 0x06ull : lane == 16 ? kPadEnd : 0ull; }
  // Four field elements (challenge limbs), in every lane; the state is unchanged.
  __device__ __forceinline__ void squeeze4_m31(uint32_t (&out)[4]) {
    const uint64_t w0 = __shfl_sync(0xffffffffu, a, 0), w1 = __shfl_sync(0xffffffffu, a, 1);
    const uint32_t c[4] = {(uint32_t)w0, (uint32_t)(w0 >> 32), (uint32_t)w1, (uint32_t)(w1 >> 32)};
    bool over = false;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      over |= c[k] >= 0xFFFFFFFEu;
      out[k] = mod_p(c[k]);
    }
    if (over) squeeze_slow(4, out);
  }
  __device__ __forceinline__ uint32_t squeeze1_m31() {
    const uint32_t c = (uint32_t)__shfl_sync(0xffffffffu, a, 0);
    uint32_t out[4] = {mod_p(c)};
    if (c >= 0xFFFFFFFEu) squeeze_slow(1, out);
    return out[0];
  }

 private:
  static __device__ __forceinline__ uint32_t mod_p(uint32_t c) {  // c < 2^32 - 2
    const uint32_t p = 2147483647u, s = (c & p) + (c >> 31);
    return s >= p ? s - p : s;
  }
  __device__ __forceinline__ void squeeze_slow(uint32_t count, uint32_t (&out)[4]) {
    __syncwarp();
    if (lane < 25) kf.col[lane] = a;
    __syncwarp();
    uint32_t o[4];
    squeeze_m31_slow(kf.col, count, o);
    for (uint32_t k = 0; k < 4; k++)
      if (k < count) out[k] = o[k];
    __syncwarp();
  }
};

// The message words of one commit-and-fold round's two frames (commitment and
// challenge), made before the root is known.
struct RoundFrames {
  uint64_t commit, challenge;
};
__device__ __forceinline__ RoundFrames circle_round_frames(uint32_t lane, uint32_t round) {
  const uint32_t c[2] = {round, 32u}, h[3] = {round, 2147483647u, 4u};
  return {frame_word<CircleFrame>(lane, 3, c), frame_word<CircleFrame>(lane, 4, h)};
}
__device__ __forceinline__ RoundFrames qm31_round_frames(uint32_t lane, uint32_t round, uint64_t in_count) {
  const uint64_t half = in_count / 2;
  const uint32_t c[6] = {round, (uint32_t)in_count, (uint32_t)(in_count >> 32), (uint32_t)half, (uint32_t)(half >> 32), 32u};
  const uint32_t h[3] = {round, 2147483647u, 4u};
  return {frame_word<Qm31Frame>(lane, 1, c), frame_word<Qm31Frame>(lane, 2, h)};
}

}  // namespace azk

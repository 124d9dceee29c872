// Host-compiled check of forms that only the kernels run (azk_keccak.cuh,
// azk_keccak_coop.cuh, azk_transcript_warp.cuh) against the CPU oracle: shortened
// digests, bit-interleaved lanes and digests, the words of the warp transcript's frames.
// Built and run by tests/test_device_forms.py.
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "azk_oracle.hpp"
#include "cuda_on_host.h"  // after the standard headers, which use some of its names
#include "azk_transcript_warp.cuh"

namespace O = azk_oracle;

#define CHECK(c, ...)                    \
  do {                                   \
    if (!(c)) {                          \
      std::fprintf(stderr, __VA_ARGS__); \
      std::fprintf(stderr, "\n");        \
      return 1;                          \
    }                                    \
  } while (0)

// The oracle's digest of lanes 0 .. bytes/8 of `l`.
static bool same(const uint64_t* l, size_t bytes, const uint64_t* d) {
  uint8_t m[136];
  std::memcpy(m, l, bytes);
  const O::Digest e = O::sha3_256(m, bytes);
  return std::memcmp(d, e.b, 32) == 0;
}

// A frame as bytes, its padded block as words.
struct Frame {
  std::vector<uint8_t> b;
  Frame(const std::string& domain, uint8_t type) {
    u32((uint32_t)domain.size());
    b.insert(b.end(), domain.begin(), domain.end());
    u32(1);
    b.push_back(type);
  }
  void u32(uint32_t v) {
    for (int k = 0; k < 4; k++) b.push_back((uint8_t)(v >> (8 * k)));
  }
  uint64_t word(uint32_t m) const {
    std::vector<uint8_t> p = b;
    p.push_back(0x06);
    p.resize(136, 0);
    p[135] |= 0x80;
    uint64_t v;
    std::memcpy(&v, p.data() + 8 * m, 8);
    return v;
  }
};
template <class F, int N>
static bool frame_is(const std::string& domain, uint8_t type, const uint32_t (&p)[N]) {
  Frame f(domain, type);
  for (uint32_t v : p) f.u32(v);
  for (uint32_t m = 0; m < 17; m++)
    if (azk::frame_word<F>(m, type, p) != f.word(m)) return false;
  return true;
}

int main() {
  std::mt19937_64 rng(7);
  for (int t = 0; t < 300; t++) {
    uint64_t l[17];
    for (auto& x : l) x = t < 4 ? (t & 1 ? ~0ull : 0ull) : rng();
    uint32_t e, o;
    azk::split64(l[0], e, o);
    for (int k = 0; k < 32; k++) CHECK(((e >> k) & 1) == ((l[0] >> (2 * k)) & 1) && ((o >> k) & 1) == ((l[0] >> (2 * k + 1)) & 1), "split bit %d", k);
    CHECK(azk::join64(e, o) == l[0], "join");
    // digests of 16 and 64 bytes and of 128 bytes (16 lanes and the suffix's)
    uint64_t a[25] = {l[0], l[1], 0x06}, d[4];
    a[16] = azk::kPadEnd;
    azk::keccak_digest<azk::kLanes16>(a, d);
    CHECK(same(l, 16, d), "digest of 16 bytes");
    uint64_t b[25] = {l[0], l[1], l[2], l[3], l[4], l[5], l[6], l[7], 0x06};
    b[16] = azk::kPadEnd;
    azk::keccak_digest<azk::kLanes64>(b, d);
    CHECK(same(l, 64, d), "digest of 64 bytes");
    uint64_t c[25] = {};
    for (int i = 0; i < 16; i++) c[i] = l[i];
    c[16] = 0x06 ^ azk::kPadEnd;
    azk::keccak_digest<azk::kLanesRate>(c, d);
    CHECK(same(l, 128, d), "digest of 128 bytes");
    // the same two in split form
    for (int pair = 0; pair < 2; pair++) {
      uint32_t se[25] = {}, so[25] = {};
      const int n = pair ? 8 : 2;
      for (int i = 0; i < n; i++) azk::split64(l[i], se[i], so[i]);
      azk::split64(0x06, se[n], so[n]);
      azk::split64(azk::kPadEnd, se[16], so[16]);
      if (pair) azk::split_round<azk::kLanes64>(se, so, 0);
      else azk::split_round<azk::kLanes16>(se, so, 0);
      const azk::SplitDigest s = azk::split_digest_rest(se, so);
      const uint64_t w[4] = {azk::join64(s.even.x, s.odd.x), azk::join64(s.even.y, s.odd.y), azk::join64(s.even.z, s.odd.z), azk::join64(s.even.w, s.odd.w)};
      CHECK(same(l, 8 * n, w), "split digest of %d bytes", 8 * n);
    }
    // padding constants of a lane pair
    for (uint32_t q = 0; q < 2; q++)
      for (uint32_t suffix : {0x06u, 0x01u}) {
        azk::split64(suffix, e, o);
        CHECK(azk::pair_suffix(suffix, q) == (q ? o : e), "suffix");
        azk::split64(azk::kPadEnd, e, o);
        CHECK(azk::pair_pad_end(q) == (q ? o : e), "end padding");
      }
    // frames of every shape the transcripts use
    uint32_t r[12];
    for (auto& x : r) x = (uint32_t)rng();
    const char *circle = "AppleZKProver.CircleFRI.PCS.V1", *qm31 = "AppleZKProver.QM31FRI.FoldChain", *sumcheck = "AppleZKProver.M31MultilinearSumcheck";
    const uint32_t p1[1] = {r[0]}, p2[2] = {r[0], r[1]}, p3[3] = {r[0], r[1], r[2]}, p4[4] = {r[0], r[1], r[2], r[3]}, p5[5] = {r[0], r[1], r[2], r[3], r[4]},
                   p6[6] = {r[0], r[1], r[2], r[3], r[4], r[5]}, p12[12] = {r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7], r[8], r[9], r[10], r[11]};
    const uint8_t type = (uint8_t)(t % 8);
    CHECK(frame_is<azk::CircleFrame>(circle, type, p1) && frame_is<azk::CircleFrame>(circle, type, p2) && frame_is<azk::CircleFrame>(circle, type, p3) &&
              frame_is<azk::CircleFrame>(circle, type, p4) && frame_is<azk::CircleFrame>(circle, type, p5),
          "circle frames");
    CHECK(frame_is<azk::Qm31Frame>(qm31, type, p3) && frame_is<azk::Qm31Frame>(qm31, type, p6), "QM31 frames");
    CHECK(frame_is<azk::SumcheckFrame>(sumcheck, type, p2) && frame_is<azk::SumcheckFrame>(sumcheck, type, p3) && frame_is<azk::SumcheckFrame>(sumcheck, type, p12),
          "sum-check frames");
    // a round's two frames, through the oracle's transcript
    const uint64_t root[4] = {rng(), rng(), rng(), rng()};
    O::Transcript ot;
    uint64_t st[25] = {};
    auto absorb = [&](auto word) {
      for (uint32_t m = 0; m < 17; m++) st[m] ^= word(m);
      azk::keccak_f1600(st);
    };
    absorb([&](uint32_t m) { return azk::circle_round_frames(m, t).commit; });
    absorb([&](uint32_t m) { return m < 4 ? root[m] : m == 4 ? 0x06ull : m == 16 ? azk::kPadEnd : 0ull; });
    absorb([&](uint32_t m) { return azk::circle_round_frames(m, t).challenge; });
    O::Digest od;
    std::memcpy(od.b, root, 32);
    O::transcript_round(ot, (uint32_t)t, od);
    for (int i = 0; i < 25; i++) CHECK(st[i] == ot.st[i], "circle round state");
  }
  std::printf("device forms ok\n");
  return 0;
}

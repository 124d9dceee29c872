// Host-compiled check of the message readers (azk_message.cuh): every message length
// at every byte alignment gives the message's words.  The exact reader reads no byte
// outside the message, the other one none outside the 4-byte units that hold message
// bytes; both only at aligned addresses.  Built and run by tests/test_message_reader.py.
#include <cstdio>
#include <cstdlib>

#include "azk_message.cuh"

static const uint8_t *lo, *hi;  // what may be read
static int outside = 0, misaligned = 0;
struct CheckedLoads {
  template <class T>
  static T load(const uint8_t* p) {
    if (p < lo || p + sizeof(T) > hi) outside++;
    if (reinterpret_cast<uintptr_t>(p) % sizeof(T)) misaligned++;
    return azk::ReadOnlyLoads::load<T>(p);
  }
};

template <bool EDGE>
static bool reads(const uint8_t* p, uint32_t len, bool aligned8) {
  lo = EDGE || aligned8 ? p : p - reinterpret_cast<uintptr_t>(p) % 4;
  hi = p + len;
  if (!EDGE && !aligned8 && len) hi += (4 - reinterpret_cast<uintptr_t>(hi) % 4) % 4;
  uint64_t want[25] = {}, a[25] = {};
  for (uint32_t k = 0; k < len; k++) want[k / 8] ^= (uint64_t)p[k] << (8 * (k % 8));
  azk::xor_message<EDGE, CheckedLoads>(a, p, len, aligned8);
  bool ok = true;
  for (int i = 0; i < 25; i++) ok &= a[i] == want[i];
  if (!aligned8) {  // words in any order, as lane pairs take them
    const azk::UnalignedWords<EDGE, CheckedLoads> u(p, len);
    for (uint32_t i = (len + 7) / 8; i-- > 0;) ok &= u.word(i, len - 8 * i < 8 ? len - 8 * i : 8) == want[i];
  }
  if (!ok || outside || misaligned)
    std::fprintf(stderr, "%s reader, offset %u, length %u, aligned8 %d: %s, %d loads outside, %d misaligned\n", EDGE ? "exact" : "unit",
                 (unsigned)(reinterpret_cast<uintptr_t>(p) % 8), len, aligned8, ok ? "words right" : "words wrong", outside, misaligned);
  return ok && !outside && !misaligned;
}

int main() {
  alignas(16) uint8_t buf[192];
  for (int i = 0; i < 192; i++) buf[i] = (uint8_t)(37 * i + 11);
  for (uint32_t off = 0; off < 8; off++)
    for (uint32_t len = 0; len <= 136; len++) {
      const uint8_t* p = buf + 16 + off;
      if (!reads<true>(p, len, false) || !reads<false>(p, len, false)) return 1;
      if (off == 0 && (!reads<true>(p, len, true) || !reads<false>(p, len, true))) return 1;
    }
  std::printf("message readers ok\n");
  return 0;
}

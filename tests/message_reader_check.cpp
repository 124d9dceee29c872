// Host-compiled check of the message readers (azk_message.cuh): every message length
// at every byte alignment gives the message's words, and of a batch's first and last
// message no byte outside it is read (of the others none outside the 4-byte units that
// hold message bytes).  Built and run by tests/test_message_reader.py.
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

int main() {
  alignas(16) uint8_t buf[192];
  for (int i = 0; i < 192; i++) buf[i] = (uint8_t)(37 * i + 11);
  for (uint32_t off = 0; off < 8; off++)
    for (uint32_t c = 0; c <= 2 * 136 + 1; c++) {
      const uint32_t len = c / 2;
      const bool edge = c % 2;
      const uint8_t* p = buf + 16 + off;
      lo = edge ? p : p - off % 4;
      hi = edge || len == 0 ? p + len : p + len + (4 - (off + len) % 4) % 4;
      uint64_t want[25] = {};
      for (uint32_t k = 0; k < len; k++) want[k / 8] ^= (uint64_t)p[k] << (8 * (k % 8));
      for (int aligned8 = 0; aligned8 <= (off == 0); aligned8++) {
        uint64_t a[25] = {};
        azk::xor_message<CheckedLoads>(a, p, len, aligned8 != 0, edge);
        for (int i = 0; i < 25; i++)
          if (a[i] != want[i] || outside || misaligned) {
            std::fprintf(stderr, "offset %u length %u aligned8 %d: lane %d, %d loads outside the message, %d misaligned\n", off, len, aligned8, i, outside,
                         misaligned);
            return 1;
          }
      }
      // words in any order, as lane pairs take them
      bool ok = true;
      azk::with_unaligned<CheckedLoads>(p, len, edge, [&](const auto& u) {
        for (uint32_t i = (len + 7) / 8; i-- > 0;) ok &= u.word(i, len - 8 * i < 8 ? len - 8 * i : 8) == want[i] && !outside && !misaligned;
      });
      if (!ok) {
        std::fprintf(stderr, "offset %u length %u: %d loads outside the message, %d misaligned\n", off, len, outside, misaligned);
        return 1;
      }
    }
  std::printf("message readers ok\n");
  return 0;
}

// First touch of large fresh result buffers (host only, no CUDA).
#pragma once
#include <algorithm>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

namespace azk {

// One byte of each page of outs[i] (bytes[i] bytes) is written, by several threads: a
// copy into fresh pages otherwise takes its page faults one after another on the calling
// thread (61 MB of proofs: 30 ms, 6 ms into touched ones).  Only a help to the copy that
// follows: where a thread cannot be had, its buffers are left to that copy.
inline void touch_pages(void* const* outs, const std::vector<uint64_t>& bytes) {
  uint64_t total = 0;
  for (uint64_t n : bytes) total += n;
  const unsigned threads = std::min(8u, std::max(1u, std::thread::hardware_concurrency() / 2));
  if (total < (4ull << 20) || threads < 2) return;
  auto touch = [&](unsigned t) {
    for (size_t i = t; i < bytes.size(); i += threads)
      for (uint64_t k = 0; k < bytes[i]; k += 4096) static_cast<volatile uint8_t*>(outs[i])[k] = 0;
  };
  std::thread pool[8];  // no allocation of its own: a thread that runs must be joined
  try {
    for (unsigned t = 1; t < threads; t++) pool[t] = std::thread(touch, t);
  } catch (const std::exception&) {
  }
  touch(0);
  for (auto& t : pool)
    if (t.joinable()) t.join();
}

}  // namespace azk

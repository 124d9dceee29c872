// Host-compiled check of touch_pages (azk_touch.h) when memory runs out at any of its
// allocations: it returns, with every thread it began joined.  Built and run by
// tests/test_touch.py.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "azk_touch.h"

static thread_local long left = -1;  // allocations this thread may still make (-1: any number)
void* operator new(size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) left--;
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main() {
  const size_t n = 64, each = 256 << 10;
  std::vector<uint64_t> bytes(n, each);
  std::vector<void*> outs;
  for (size_t i = 0; i < n; i++) outs.push_back(std::malloc(each));
  for (long k = 0; k < 24; k++) {
    left = k;
    azk::touch_pages(outs.data(), bytes);
    left = -1;
  }
  azk::touch_pages(outs.data(), bytes);
  for (void* p : outs)
    for (size_t k = 0; k < each; k += 4096)
      if (static_cast<uint8_t*>(p)[k] != 0) return 1;
  std::printf("touch ok\n");
  return 0;
}

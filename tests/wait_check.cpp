// Host-compiled check of the waits and turns (azk_wait.h): no more threads spin at a
// time than there are places, the others sleep between polls soon after they begin to
// wait, places are given back, also when a poll throws.  Built and run by
// tests/test_wait.py.
#include <cstdio>
#include <stdexcept>
#include <vector>

#include "azk_wait.h"

#define CHECK(c, what)                       \
  do {                                       \
    if (!(c)) {                              \
      std::fprintf(stderr, "%s\n", what);    \
      return 1;                              \
    }                                        \
  } while (0)

int main() {
  using namespace azk;
  // one place, taken: polls 8 times, then sleeps that grow
  {
    SpinPlaces places(1);
    SpinPlace held(places, true);
    CHECK(held.at && places.taken == 1, "the first thread spins");
    std::vector<uint32_t> slept;
    int polls = 0;
    poll_until([&] { return ++polls > 80; }, [&](uint32_t us) { slept.push_back(us); }, false, places);
    CHECK(polls == 81 && slept.size() == 72, "a thread without a place sleeps after 8 polls");
    CHECK(slept.front() == 20 && slept[20] == 50 && slept.back() == 160, "its sleeps grow from 20 to 160 us");
    CHECK(places.taken == 1, "it takes no place");
  }
  // a free place: spins, then sleeps of 20 us
  {
    SpinPlaces places(1);
    std::vector<uint32_t> slept;
    const auto t0 = std::chrono::steady_clock::now();
    int after = 0;
    poll_until([&] { return !slept.empty() && ++after > 3; }, [&](uint32_t us) { slept.push_back(us); }, false, places);
    CHECK(std::chrono::steady_clock::now() - t0 >= std::chrono::milliseconds(5), "a thread with a place spins for 5 ms");
    CHECK(slept.back() == 20 && places.taken == 0, "and then sleeps 20 us at a time, its place given back");
  }
  // shared host and a poll that throws
  {
    SpinPlaces places(4);
    std::vector<uint32_t> slept;
    int polls = 0;
    poll_until([&] { CHECK(places.taken == 0, "a shared thread takes no place"); return (int)(++polls > 20); }, [&](uint32_t us) { slept.push_back(us); }, true,
               places);
    CHECK(slept.size() == 12, "a shared thread sleeps");
    polls = 0;
    try {
      poll_until([&]() -> bool { if (++polls > 4) throw std::runtime_error("x"); return false; }, [](uint32_t) {}, false, places);
      return 1;
    } catch (const std::runtime_error&) {
    }
    CHECK(places.taken == 0, "a place is given back when a poll throws");
  }
  // many threads: all but the two with places sleep at once, those after their 5 ms
  {
    SpinPlaces places(2);
    std::atomic<int> sleeping{0};
    std::atomic<bool> go{false};
    std::vector<std::thread> pool;
    for (int i = 0; i < 8; i++)
      pool.emplace_back([&] {
        bool counted = false;
        poll_until([&] { return go.load(); },
                   [&](uint32_t us) {
                     if (!counted) sleeping++;
                     counted = true;
                     std::this_thread::sleep_for(std::chrono::microseconds(us));
                   },
                   false, places);
      });
    while (sleeping < 8) std::this_thread::yield();  // the two that spun sleep after 5 ms
    go = true;
    for (auto& t : pool) t.join();
    CHECK(places.taken == 0, "places add up");
  }
  // turns are taken in the order of arrival, also against a thread that comes back at once
  {
    Turns turns;
    std::vector<int> order;
    std::vector<std::thread> pool;
    {
      Turns::Turn held(turns);
      for (int i = 0; i < 6; i++) {
        pool.emplace_back([&, i] {
          Turns::Turn t(turns);
          order.push_back(i);
        });
        for (;;) {  // the thread has its place in the line
          std::lock_guard<std::mutex> lk(turns.mu);
          if (turns.next == (uint64_t)i + 2) break;
        }
      }
    }
    { Turns::Turn back(turns); order.push_back(6); }
    for (auto& t : pool) t.join();
    CHECK((order == std::vector<int>{0, 1, 2, 3, 4, 5, 6}), "turns in the order of arrival");
  }
  CHECK(SpinPlaces::usable_cores() >= 1 && SpinPlaces::process().most == SpinPlaces::usable_cores() / 2, "half of the host's cores");
  std::printf("waits ok\n");
  return 0;
}

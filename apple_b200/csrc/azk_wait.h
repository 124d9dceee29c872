// How a thread waits for the device by polling (host only, no CUDA).
//
// A caller's own thread spins for up to 5 ms, as CUDA's own synchronisation does (a
// sleep of 20 us lasts about 75 with the kernel's timer slack: 25 to 100 us on calls
// whose device time is 30 to 250), and sleeps between polls after that.  At most half
// of the host's cores spin at a time: a thread that finds them taken (a program with
// as many proving threads as cores, or one core) polls a few times and then sleeps
// growing from 20 to 160 us, and so do the server's workers and lane threads.
#pragma once
#include <sched.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <thread>

namespace azk {

// The places for spinning threads of a process.
struct SpinPlaces {
  std::atomic<int> taken{0};
  int most;
  explicit SpinPlaces(int n) : most(n) {}
  static int usable_cores() {
    cpu_set_t set;
    if (sched_getaffinity(0, sizeof(set), &set) == 0) return CPU_COUNT(&set);
    const unsigned n = std::thread::hardware_concurrency();
    return n ? (int)n : 1;
  }
  static SpinPlaces& process() {
    static SpinPlaces places(usable_cores() / 2);
    return places;
  }
};
struct SpinPlace {
  SpinPlaces* at;
  SpinPlace(SpinPlaces& p, bool wanted) : at(wanted ? &p : nullptr) {
    if (at && at->taken.fetch_add(1, std::memory_order_relaxed) >= at->most) release();
  }
  ~SpinPlace() { release(); }
  SpinPlace(const SpinPlace&) = delete;
  SpinPlace& operator=(const SpinPlace&) = delete;
  void release() {
    if (at) at->taken.fetch_sub(1, std::memory_order_relaxed);
    at = nullptr;
  }
};

// Poll done() until it holds; sleep(microseconds) between polls.  shared_host: never
// spin.
template <class Done, class Sleep>
void poll_until(Done done, Sleep sleep, bool shared_host, SpinPlaces& places) {
  if (done()) return;
  const auto t0 = std::chrono::steady_clock::now();
  SpinPlace place(places, !shared_host);
  const bool spun = place.at != nullptr;
  for (uint32_t k = 1; !done(); k++) {
    if (place.at) {
      if (std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(5)) place.release();
    } else if (spun) {
      sleep(20u);
    } else if (k >= 8) {
      sleep(k < 24 ? 20u : k < 48 ? 50u : 160u);
    }
  }
}

// One thread at a time, in the order they came (a std::mutex lets a thread that returns
// at once pass those that wait).
struct Turns {
  struct Turn {
    Turns& of;
    explicit Turn(Turns& t) : of(t) {
      std::unique_lock<std::mutex> lk(of.mu);
      const uint64_t mine = of.next++;
      of.moved.wait(lk, [&] { return of.now == mine; });
    }
    ~Turn() {
      std::lock_guard<std::mutex> lk(of.mu);
      of.now++;
      if (of.now != of.next) of.moved.notify_all();
    }
    Turn(const Turn&) = delete;
    Turn& operator=(const Turn&) = delete;
  };
  std::mutex mu;
  std::condition_variable moved;
  uint64_t next = 0, now = 0;
};

}  // namespace azk

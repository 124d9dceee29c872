// Host-side runtime shared by the C-ABI translation units: context, error
// handling, device buffers, domain-table cache and the work-list builders.
#pragma once
#include <cuda_runtime.h>

#if defined(__SSE2__) && !defined(__CUDA_ARCH__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <array>
#include <chrono>
#include <cstring>
#include <initializer_list>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "../../include/azk_cuda.h"
#include "azk_internal.h"
#include "azk_wait.h"

// Page-locked memory that results cross to the host through, and an event for each half
// of it.
struct azk_landing {
  void* p = nullptr;
  uint64_t n = 0;
  cudaEvent_t half[2] = {nullptr, nullptr};
  azk_landing() = default;
  azk_landing(const azk_landing&) = delete;
  azk_landing& operator=(const azk_landing&) = delete;
  ~azk_landing() {
    if (p) cudaFreeHost(p);
    for (auto& e : half)
      if (e) cudaEventDestroy(e);
  }
};

struct azk_ctx {
  int device = 0;
  int sm_count = 0;
  int cc_major = 0, cc_minor = 0;
  uint64_t total_mem = 0;
  cudaStream_t stream = nullptr;
  std::mutex mu;
  std::string last_error;
  struct Domain {
    uint32_t* tw = nullptr;  // N - 1 stage twiddles, then (at tw + N) the same doubled
    uint32_t* inv = nullptr;
  };
  std::map<uint32_t, Domain> domains;
  // Scratch of azk_sumcheck_prove for tables of at most 2^kSumcheckKeptLog words (8.4
  // MB on the device, 4.2 MB page-locked), used under `mu`, freed with the context;
  // larger tables take their own for the call.
  static constexpr uint32_t kSumcheckKeptLog = 20;
  void* sumcheck_dev = nullptr;
  void* sumcheck_pin = nullptr;
  uint64_t sumcheck_dev_bytes = 0, sumcheck_pin_bytes = 0;
  // Landings that no call is using, at most kLandingsKept (of at most 2 MB each), freed
  // with the context.
  static constexpr size_t kLandingsKept = 32;
  std::mutex landing_mu;
  std::vector<std::unique_ptr<azk_landing>> landings;
  azk::Turns upload_turns;  // of large copies from pageable memory
};

namespace azk {

struct Error {
  azk_status code;
  std::string msg;
};

[[noreturn]] inline void fail(azk_status code, const std::string& msg) { throw Error{code, msg}; }
inline void require(bool ok, azk_status code, const std::string& msg) {
  if (!ok) fail(code, msg);
}
inline void layout(bool ok, const char* what = "The provided input bytes do not match the declared count/stride/length layout.") {
  if (!ok) fail(AZK_ERR_INVALID_INPUT_LAYOUT, what);
}
// Whether all `n` words are canonical M31 values (below 2^31 - 1): one
// branch-free pass that the host compiler vectorises (a 4 MiB table in about
// 0.1 ms, against about 1 ms for a compare-and-branch per word).
inline bool all_canonical(const uint32_t* w, uint64_t n) {
  uint32_t bad = 0;
  for (uint64_t i = 0; i < n; i++) bad |= (uint32_t)(w[i] >= 2147483647u);
  return bad == 0;
}

#define AZK_CU(expr)                                                                                   \
  do {                                                                                                 \
    cudaError_t azk_e_ = (expr);                                                                       \
    if (azk_e_ != cudaSuccess)                                                                         \
      ::azk::fail(AZK_ERR_COMMAND_EXECUTION_FAILED, std::string(#expr) + ": " + cudaGetErrorString(azk_e_)); \
  } while (0)

void set_error(const azk_ctx* ctx, const std::string& msg);

template <class F>
azk_status guarded(const azk_ctx* ctx, F&& f) {
  try {
    f();
    return AZK_OK;
  } catch (const Error& e) {
    set_error(ctx, e.msg);
    return e.code;
  } catch (const std::bad_alloc&) {
    set_error(ctx, "host allocation failed");
    return AZK_ERR_FAILED_TO_CREATE_BUFFER;
  } catch (const std::exception& e) {
    set_error(ctx, e.what());
    return AZK_ERR_COMMAND_EXECUTION_FAILED;
  }
}

inline bool is_pow2(uint64_t v) { return v && !(v & (v - 1)); }
inline uint32_t ilog2(uint64_t v) {
  uint32_t r = 0;
  while (v > 1) { v >>= 1; r++; }
  return r;
}
inline uint64_t align_up(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }

// Owning device allocation.
struct DevBuf {
  void* p = nullptr;
  uint64_t bytes = 0;
  DevBuf() = default;
  explicit DevBuf(uint64_t n, const char* label = "buffer") { alloc(n, label); }
  void alloc(uint64_t n, const char* label = "buffer") {
    release();
    if (n == 0) n = 16;
    cudaError_t e = cudaMalloc(&p, n);
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();
      fail(AZK_ERR_FAILED_TO_CREATE_BUFFER, std::string("Failed to create device buffer '") + label + "' of length " + std::to_string(n));
    }
    bytes = n;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  ~DevBuf() { release(); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes) {
    o.p = nullptr;
    o.bytes = 0;
  }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      bytes = o.bytes;
      o.p = nullptr;
      o.bytes = 0;
    }
    return *this;
  }
  template <class T>
  T* as() const { return reinterpret_cast<T*>(p); }
};

// Bump allocator over one device allocation (the reference's ResidencyArena,
// Planner/ResidencyArena.swift:36-92: 256-byte aligned slices).
struct Arena {
  DevBuf buf;
  uint64_t used = 0;
  std::vector<std::pair<uint64_t, uint64_t>> plan;  // (offset, bytes) reservations before alloc
  uint64_t reserve(uint64_t bytes) {
    uint64_t off = align_up(used, 256);
    used = off + (bytes ? bytes : 16);
    return off;
  }
  void commit(const char* label) { buf.alloc(used, label); }
  template <class T>
  T* at(uint64_t off) const { return reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(buf.p) + off); }
};

struct Timer {
  std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
  double seconds() const { return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); }
  uint64_t ns() const { return (uint64_t)std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now() - t0).count(); }
};

// Threads that share the host's cores with many others (the server's workers and
// lane threads) set this for themselves; their waits then sleep early.
inline thread_local bool t_shared_host = false;

// Wait for an event by polling it (azk_wait.h).
// Not cudaEventSynchronize on a blocking-sync event, which sleeps until the
// driver's completion interrupt: with the server's 32 workers waiting that way at
// once, the device stopped starting work for 40-80 ms about every 2 s.
inline void wait_event(cudaEvent_t e) {
  poll_until(
      [e] {
        const cudaError_t q = cudaEventQuery(e);
        if (q != cudaErrorNotReady) AZK_CU(q);
        return q == cudaSuccess;
      },
      [](uint32_t us) { std::this_thread::sleep_for(std::chrono::microseconds(us)); }, t_shared_host, SpinPlaces::process());
}

// Wait for everything queued on a stream (wait_event on a per-thread event).
inline void sync_stream(cudaStream_t s) {
  struct Ev {
    cudaEvent_t e = nullptr;
    int dev = -1;
    ~Ev() {
      if (e) cudaEventDestroy(e);
    }
  };
  thread_local Ev ev;
  int dev = 0;
  AZK_CU(cudaGetDevice(&dev));
  if (!ev.e || ev.dev != dev) {
    if (ev.e) cudaEventDestroy(ev.e);
    ev.e = nullptr;
    AZK_CU(cudaEventCreateWithFlags(&ev.e, cudaEventDisableTiming));
    ev.dev = dev;
  }
  AZK_CU(cudaEventRecord(ev.e, s));
  wait_event(ev.e);
}

// A thread's timing events on its current device, kept from one timed region to the
// next (creating and destroying a pair costs about as much as two launches); nested
// regions take further pairs.  At most eight pairs, destroyed with the thread.
struct TimingEvents {
  struct Pair {
    cudaEvent_t a = nullptr, b = nullptr;
    int dev = -1;
    bool busy = false;
  };
  Pair pair[8];
  ~TimingEvents() {
    for (auto& p : pair) {
      if (p.a) cudaEventDestroy(p.a);
      if (p.b) cudaEventDestroy(p.b);
    }
  }
  static TimingEvents& mine() {
    thread_local TimingEvents t;
    return t;
  }
  // A free pair of the current device (an unused slot is filled), or null.
  Pair* take() {
    int dev = 0;
    AZK_CU(cudaGetDevice(&dev));
    Pair* empty = nullptr;
    for (auto& p : pair) {
      if (p.busy) continue;
      if (p.a && p.b && p.dev == dev) {
        p.busy = true;
        return &p;
      }
      if (!p.a && !empty) empty = &p;
    }
    if (!empty) return nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    AZK_CU(cudaEventCreate(&a));
    const cudaError_t e = cudaEventCreate(&b);
    if (e != cudaSuccess) cudaEventDestroy(a);
    AZK_CU(e);
    empty->a = a;
    empty->b = b;
    empty->dev = dev;
    empty->busy = true;
    return empty;
  }
};

// CUDA events around a region of one stream; used and destroyed by one thread.
struct GpuTimer {
  cudaEvent_t a = nullptr, b = nullptr;
  cudaStream_t s;
  TimingEvents::Pair* kept = nullptr;
  bool owns = false;
  explicit GpuTimer(cudaStream_t st) : s(st) {
    kept = TimingEvents::mine().take();
    if (kept) {
      a = kept->a;
      b = kept->b;
    } else {
      owns = true;
      AZK_CU(cudaEventCreate(&a));
      AZK_CU(cudaEventCreate(&b));
    }
    AZK_CU(cudaEventRecord(a, s));
  }
  // With events the caller keeps.
  GpuTimer(cudaStream_t st, cudaEvent_t ea, cudaEvent_t eb) : a(ea), b(eb), s(st) { AZK_CU(cudaEventRecord(a, s)); }
  GpuTimer(const GpuTimer&) = delete;
  GpuTimer& operator=(const GpuTimer&) = delete;
  void stop() { AZK_CU(cudaEventRecord(b, s)); }
  double seconds() {
    float ms = 0;
    wait_event(b);
    AZK_CU(cudaEventElapsedTime(&ms, a, b));
    return ms / 1000.0;
  }
  ~GpuTimer() {
    if (kept) kept->busy = false;
    if (!owns) return;
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
  }
};

// Page-locked host memory kept for the owner's lifetime: small uploads and
// readbacks go through it rather than through pageable memory, which the driver
// stages through buffers shared by every thread of the process.
struct HostPinned {
  void* p = nullptr;
  size_t n = 0;
  HostPinned() = default;
  HostPinned(const HostPinned&) = delete;
  HostPinned& operator=(const HostPinned&) = delete;
  void* ensure(size_t bytes) {
    if (bytes > n) {
      if (p) cudaFreeHost(p);
      p = nullptr;
      n = 0;
      AZK_CU(cudaHostAlloc(&p, bytes, cudaHostAllocDefault));
      n = bytes;
    }
    return p;
  }
  ~HostPinned() {
    if (p) cudaFreeHost(p);
  }
};

// Results on their way to a caller's memory: the copies are queued on `s`, the stream
// is waited for, check() may refuse the results, and `dst` (null: skipped) is written.
// They cross through page-locked memory that the context keeps, at once up to
// kLandingPiece, in pieces above.  A copy to pageable memory holds a lock
// of the driver while it waits, and the driver does not hand that lock out in turn: with
// a dozen threads in calls that end in such copies, some threads got no call through until
// the others stopped (32 threads with a 2^14 prover each: all but six, 7,900 proofs/s in
// all against 19,700 so).
struct HostResult {
  void* dst;
  const void* src;
  uint64_t bytes;
};
static constexpr uint64_t kLandingBytes = 2ull << 20, kLandingPiece = kLandingBytes / 2;
// One of the context's landings, for the duration of a call.
struct LandingLease {
  azk_ctx* ctx;
  std::unique_ptr<azk_landing> l;
  LandingLease(azk_ctx* c, uint64_t bytes) : ctx(c) {
    {
      // the smallest one that is large enough, else the largest
      std::lock_guard<std::mutex> lk(c->landing_mu);
      auto& v = c->landings;
      size_t best = v.size();
      for (size_t i = 0; i < v.size(); i++) {
        const bool fits = v[i]->n >= bytes;
        if (best == v.size() || (fits ? v[best]->n < bytes || v[i]->n < v[best]->n : v[best]->n < bytes && v[i]->n > v[best]->n)) best = i;
      }
      if (best < v.size()) {
        l = std::move(v[best]);
        v[best] = std::move(v.back());
        v.pop_back();
      }
    }
    if (!l) l = std::make_unique<azk_landing>();
    if (l->n >= bytes) return;
    uint64_t m = 16384;
    while (m < bytes) m *= 2;
    if (l->p) cudaFreeHost(l->p);
    l->p = nullptr;
    l->n = 0;
    if (cudaHostAlloc(&l->p, m, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      l->p = nullptr;
    } else {
      l->n = m;
    }
  }
  ~LandingLease() {
    std::lock_guard<std::mutex> lk(ctx->landing_mu);
    if (l->p && ctx->landings.size() < azk_ctx::kLandingsKept) ctx->landings.push_back(std::move(l));  // reserved by azk_ctx_create
  }
  LandingLease(const LandingLease&) = delete;
  LandingLease& operator=(const LandingLease&) = delete;
  // Page-locked bytes, or null where there are none to be had.
  uint8_t* bytes() const { return static_cast<uint8_t*>(l->p); }
  cudaEvent_t* halves() const {
    for (auto& e : l->half)
      if (!e) AZK_CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return l->half;
  }
};
// Waits for the stream unless told that it is idle: an error must not leave copies in
// flight into a landing that the next call takes.
struct SettleStream {
  cudaStream_t s;
  bool idle = false;
  explicit SettleStream(cudaStream_t st) : s(st) {}
  ~SettleStream() {
    if (!idle) cudaStreamSynchronize(s);
  }
  SettleStream(const SettleStream&) = delete;
  SettleStream& operator=(const SettleStream&) = delete;
};
// memcpy of a piece of a large result, past the caches where the host has such stores:
// lines of the destination are not read first (a 2^20 codeword of 16 MB to the host: 2.66
// ms a call with memcpy, 2.30 so, 2.32 by the driver's own pageable copy).
inline void copy_past_caches(uint8_t* dst, const uint8_t* src, uint64_t n) {
#if defined(__SSE2__) && !defined(__CUDA_ARCH__)
  const uint64_t head = std::min<uint64_t>((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15, n);
  std::memcpy(dst, src, head);
  uint64_t k = head;
  for (; k + 64 <= n; k += 64) {
    const __m128i* f = reinterpret_cast<const __m128i*>(src + k);
    __m128i* t = reinterpret_cast<__m128i*>(dst + k);
    const __m128i a = _mm_loadu_si128(f), b = _mm_loadu_si128(f + 1), c = _mm_loadu_si128(f + 2), d = _mm_loadu_si128(f + 3);
    _mm_stream_si128(t, a);
    _mm_stream_si128(t + 1, b);
    _mm_stream_si128(t + 2, c);
    _mm_stream_si128(t + 3, d);
  }
  _mm_sfence();
  std::memcpy(dst + k, src + k, n - k);
#else
  std::memcpy(dst, src, n);
#endif
}
// Host memory that a copy reaches without the driver's staging.
inline bool page_locked(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}
static constexpr uint64_t kLandingSmall = 32ull << 10;  // results up to here are not worth the question
template <class Check>
void read_back(azk_ctx* ctx, cudaStream_t s, const HostResult* results, size_t count, Check check) {
  // results that need a landing, and those for page-locked memory of the caller's, which
  // are copied straight to it once check() has passed (it may run twice then)
  std::optional<LandingLease> lease;  // given back after `settle`
  SettleStream settle(s);
  std::vector<HostResult> r, straight;
  uint64_t total = 0;
  for (size_t i = 0; i < count; i++) {
    if (!results[i].dst || !results[i].bytes) continue;
    const bool locked = results[i].bytes > kLandingSmall && page_locked(results[i].dst);
    (locked ? straight : r).push_back(results[i]);
    if (!locked) total += align_up(results[i].bytes, 16);
  }
  const size_t n = r.size();
  if (!straight.empty() || n == 0) {
    sync_stream(s);
    check();
    for (const HostResult& h : straight) AZK_CU(cudaMemcpyAsync(h.dst, h.src, h.bytes, cudaMemcpyDeviceToHost, s));
    if (n == 0) {
      if (!straight.empty()) sync_stream(s);
      settle.idle = true;
      return;
    }
  }
  lease.emplace(ctx, total <= kLandingPiece ? total : kLandingBytes);
  uint8_t* const landing = lease->bytes();
  if (landing && total <= kLandingPiece) {
    uint64_t at = 0;
    for (size_t i = 0; i < n; i++) {
      AZK_CU(cudaMemcpyAsync(landing + at, r[i].src, r[i].bytes, cudaMemcpyDeviceToHost, s));
      at += align_up(r[i].bytes, 16);
    }
    sync_stream(s);
    settle.idle = true;
    check();
    at = 0;
    for (size_t i = 0; i < n; i++) {
      std::memcpy(r[i].dst, landing + at, r[i].bytes);
      at += align_up(r[i].bytes, 16);
    }
    return;
  }
  if (!landing) {
    sync_stream(s);
    check();
    for (const HostResult& h : r) AZK_CU(cudaMemcpyAsync(h.dst, h.src, h.bytes, cudaMemcpyDeviceToHost, s));
    sync_stream(s);
    settle.idle = true;
    return;
  }
  // In pieces, one copied out while the next one is in flight; small ones where the
  // first one's way and the last one's copying would otherwise be most of the time.
  const uint64_t most = total >= 4 * kLandingPiece ? kLandingPiece : kLandingPiece / 4;
  cudaEvent_t* const half = lease->halves();
  struct Part {
    uint8_t* dst;
    uint64_t at, bytes;
  };
  std::vector<Part> part[2];  // what a half holds: the end of one result, small ones whole, the start of another
  uint64_t used[2] = {0, 0};
  bool checked = false;
  auto finish = [&](uint32_t h) {
    if (!used[h]) return;
    wait_event(half[h]);
    if (!checked) check();
    checked = true;
    for (const Part& q : part[h]) copy_past_caches(q.dst, landing + h * kLandingPiece + q.at, q.bytes);
    part[h].clear();
    used[h] = 0;
  };
  uint32_t h = 0;
  for (size_t i = 0; i < n; i++) {
    for (uint64_t at = 0; at < r[i].bytes;) {
      const uint64_t bytes = std::min(r[i].bytes - at, most - used[h]);
      AZK_CU(cudaMemcpyAsync(landing + h * kLandingPiece + used[h], static_cast<const uint8_t*>(r[i].src) + at, bytes, cudaMemcpyDeviceToHost, s));
      part[h].push_back({static_cast<uint8_t*>(r[i].dst) + at, used[h], bytes});
      used[h] += align_up(bytes, 16);
      at += bytes;
      if (used[h] < most && !(i + 1 == n && at == r[i].bytes)) continue;
      AZK_CU(cudaEventRecord(half[h], s));
      h ^= 1;
      finish(h);
    }
  }
  finish(h);
  finish(h ^ 1);
  settle.idle = true;  // every piece was waited for
}
inline void read_back(azk_ctx* ctx, cudaStream_t s, std::initializer_list<HostResult> r) { read_back(ctx, s, r.begin(), r.size(), [] {}); }

// A caller's input to the device, `src` read before this returns.  The driver's copy from
// pageable memory takes the same lock, so large ones go to it one thread at a time, in the
// order they came (twelve threads with 4 MB of coefficients each: without turns one got a
// single call through in 0.6 s).  Staging them here instead, through page-locked pieces,
// made a call alone 3 to 19 % slower.
static constexpr uint64_t kUploadSmall = 64ull << 10;
inline void upload(azk_ctx* ctx, cudaStream_t s, void* dst, const void* src, uint64_t bytes) {
  if (bytes == 0) return;
  std::optional<Turns::Turn> turn;
  if (bytes > kUploadSmall && !page_locked(src)) turn.emplace(ctx->upload_turns);
  AZK_CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
}

inline void fill_stats(azk_stats* st, const Timer& t, uint64_t submit_ns, double gpu_s) {
  if (!st) return;
  st->cpu_wall_s = t.seconds();
  st->gpu_s = gpu_s;
  st->cpu_submit_ns = submit_ns;
}

// Resident entry points take (device pointer, byte offset) pairs.  This checks
// that [p + off, p + off + bytes) lies inside the one device allocation containing
// p + off (the reference's buffer-length check, e.g. QM31FRIFold.swift:1236-1244),
// failing with AZK_ERR_INVALID_INPUT_LAYOUT otherwise or when the address is not
// device memory.
void require_device_range(const void* p, uint64_t off, uint64_t bytes);
// Two byte ranges of device memory overlap (the reference's rangesOverlap on one
// buffer, QM31FRIFold.swift:1280-1294; distinct allocations never overlap).
inline bool ranges_overlap(const void* a, uint64_t aoff, uint64_t abytes, const void* b, uint64_t boff, uint64_t bbytes) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a) + aoff, y = reinterpret_cast<uintptr_t>(b) + boff;
  return x < y + bbytes && y < x + abytes;
}

// Domain tables of size 2^logn, materialised once per context.
const azk_ctx::Domain& domain_tables(azk_ctx* ctx, uint32_t logn);

// Resolved hashing schedule.
struct Sched {
  uint32_t tile_log = 12;
  uint32_t group_log = 12;
  uint32_t threads = 256;
  bool graph = true;
  uint8_t layer_tile[32] = {0};
  uint16_t layer_threads[32] = {0};
  bool persistent_trees = false;
};
// A schedule with no treelet depth and no layer table takes `defaults` (a tuned
// per-layer table from azk_tuned.h) when one is given, and with no thread count
// and no per-layer threads `default_threads` likewise.
Sched resolve_schedule(const azk_schedule* s, const uint8_t* defaults = nullptr, const uint16_t* default_threads = nullptr);
// Threads per CTA of the commit kernel for a layer of 2^logn leaves.
inline uint32_t tree_threads(const Sched& s, uint32_t logn) { return (logn < 32 && s.layer_threads[logn]) ? s.layer_threads[logn] : s.threads; }
// Tile depth used for a tree of 2^logn leaves under a schedule (per-layer table
// first, then the global depth), clamped to [1, logn].
inline uint32_t tree_tile_log(const Sched& s, uint32_t logn) {
  uint32_t t = (logn < 32 && s.layer_tile[logn]) ? s.layer_tile[logn] : s.tile_log;
  if (t > logn) t = logn;
  if (t == 0 && logn > 0) t = 1;
  return t;
}

// FFT work for a set of transforms: one FftJob per (transform, pass); passes of
// all transforms are aligned so every transform's last (low-stage) pass runs at
// the final step.  Inside a step the work items are grouped by pass kernel
// (FftKind: QM31 tiles, small one-limb transforms, one-limb tiles, bulk-copied
// one-limb low passes), each group one contiguous range and one launch.
// Transforms flagged `narrow` (inputs known to be lifted M31 polynomials) take the
// one-limb kernels.
struct FftPlan {
  std::vector<FftJob> jobs;
  std::vector<uint2> work;  // all steps, step-major, kind-major, transform-contiguous
  std::vector<std::array<uint64_t, kFftKinds>> part_off, part_cnt;  // per step and kind
  std::vector<uint8_t> narrow;                                      // per transform
  std::vector<std::vector<std::pair<uint64_t, uint64_t>>> inst_range;  // [step][transform] -> (offset, count)
  std::vector<std::vector<uint8_t>> inst_kind;                         // [step][transform] -> FftKind
  DevBuf d_jobs, d_work;
  DevBuf d_status;  // raised by a pass kernel whose bounded wait ran out
  size_t steps() const { return part_off.size(); }
  void build(const std::vector<FftJob>& transforms, const std::vector<uint8_t>& narrow_flags = {});
  void upload(cudaStream_t s);
  void launch_step(size_t step, cudaStream_t s) const;
  void launch_step_for(size_t step, size_t t, cudaStream_t s) const;
  void launch_all(cudaStream_t s) const {
    for (size_t k = 0; k < steps(); k++) launch_step(k, s);
  }
  // Queue the readback of the status word into `host_word` (page-locked), and, once
  // the stream has finished, fail with AZK_ERR_DEVICE_TIMEOUT (clearing the flag) when
  // a pass kernel gave up waiting for its tile copies.
  void queue_status(cudaStream_t s, uint32_t* host_word) const;
  void check_status(cudaStream_t s, const uint32_t* host_word) const;
};

// Monomial -> interleaved circle FFT-basis coefficients, host-side like the
// reference's CircleCodewordPlan (CircleCodeword.swift:100-127, 187-263).
std::vector<uint32_t> fft_basis_from_monomials(uint32_t logn, const uint32_t* x, uint64_t nx, const uint32_t* y, uint64_t ny);

}  // namespace azk

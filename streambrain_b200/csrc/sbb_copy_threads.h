// memcpy by several threads, for the copies between pageable and pinned host memory (host code only).
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include <sched.h>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace sbb {

// One job at a time, cut into pieces that the caller and the workers claim one by one: whoever is late, for a worker still
// waking up, finds nothing left.  Workers spin for 200 us after a job (a copy is a series of jobs) before they sleep.  Up to 11
// of them, and no more than the process's share of three quarters of the machine's hardware threads leaves beside the caller.
class CopyThreads {
 public:
  static CopyThreads &get() {
    static CopyThreads t;
    return t;
  }
  // `past_cache`: large copies are written past the caches, for a destination that nobody reads soon (without reading it
  // first, as a store to a line that is not in the cache does: 153 against 66 GB/s by eight threads).
  void copy(void *dst, const void *src, size_t bytes, bool past_cache = false) {
    past_cache = past_cache && bytes >= kPastCache;
    if (bytes <= kAlone || workers_.empty() || !mutex_.try_lock()) {   // (busy with another thread's job)
      move(static_cast<char *>(dst), static_cast<const char *>(src), bytes, past_cache);
      return;
    }
    const uint32_t pieces = (uint32_t)((bytes + kPiece - 1) / kPiece);
    const uint64_t generation = (next_.load(std::memory_order_relaxed) >> 32) + 1;
    dst_.store(static_cast<char *>(dst), std::memory_order_relaxed);
    src_.store(static_cast<const char *>(src), std::memory_order_relaxed);
    bytes_.store(bytes, std::memory_order_relaxed);
    past_cache_.store(past_cache, std::memory_order_relaxed);
    done_.store(0, std::memory_order_relaxed);
    next_.store(generation << 32, std::memory_order_release);
    if (asleep_.load() > 0) {
      { std::lock_guard<std::mutex> l(sleep_mutex_); }
      wake_.notify_all();
    }
    while (take_piece()) {
    }
    while (done_.load(std::memory_order_acquire) < pieces) std::this_thread::yield();
    next_.store(generation << 32 | kClosed, std::memory_order_release);   // before the fields change again
    mutex_.unlock();
  }

 private:
  static constexpr size_t kPiece = 32 << 10;   // (half a microsecond to copy in cache, two from memory)
  static constexpr size_t kAlone = 128 << 10;   // up to here the workers cost more than they save (84 KB: 4 us)
  static constexpr size_t kPastCache = 512 << 10;
  static constexpr uint32_t kClosed = 0xFFFFFFFFu;
  static void move(char *dst, const char *src, size_t bytes, bool past_cache) {
#ifdef __SSE2__
    if (past_cache) {
      const size_t head = -reinterpret_cast<uintptr_t>(dst) & 15;
      if (head < bytes) {
        std::memcpy(dst, src, head);
        dst += head, src += head, bytes -= head;
        for (; bytes >= 64; dst += 64, src += 64, bytes -= 64) {
          const __m128i *s = reinterpret_cast<const __m128i *>(src);
          __m128i *d = reinterpret_cast<__m128i *>(dst);
          const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
          _mm_stream_si128(d, a), _mm_stream_si128(d + 1, b), _mm_stream_si128(d + 2, c), _mm_stream_si128(d + 3, e);
        }
        _mm_sfence();   // before the piece counts as done
      }
    }
#endif
    std::memcpy(dst, src, bytes);
  }
  // Hardware threads this process may count on: those it is bound to, and an even part of the machine's where a launcher says
  // that it started several processes here (eight of them with eleven spinning threads each would take the cores from one another).
  static unsigned share() {
    unsigned n = std::thread::hardware_concurrency();
    const char *e = std::getenv("LOCAL_WORLD_SIZE");
    const long processes = e != nullptr ? std::strtol(e, nullptr, 10) : 1;
    if (processes > 1) n = (unsigned)(n / processes);
    cpu_set_t bound;
    if (sched_getaffinity(0, sizeof(bound), &bound) == 0 && (unsigned)CPU_COUNT(&bound) < n) n = (unsigned)CPU_COUNT(&bound);
    return n;
  }
  CopyThreads() {
    unsigned n = share() / 4 * 3;
    if (n > 12) n = 12;
    try {   // (a process may be out of threads or memory: the callers then copy with those there are, or by themselves)
      for (unsigned k = 1; k < n; ++k) workers_.emplace_back([this] { work(); });
    } catch (const std::exception &) {
    }
  }
  ~CopyThreads() {
    {
      std::lock_guard<std::mutex> l(sleep_mutex_);
      stop_.store(true);
    }
    wake_.notify_all();
    for (auto &w : workers_) w.join();
  }
  // The fields change only while the job is closed, and a claim fails when the job number or its next piece has changed
  // since they were read: fields read before a successful claim belong to the claimed job.
  bool take_piece() {
    uint64_t v = next_.load(std::memory_order_acquire);
    while (true) {
      char *dst = dst_.load(std::memory_order_relaxed);
      const char *src = src_.load(std::memory_order_relaxed);
      const bool past_cache = past_cache_.load(std::memory_order_relaxed);
      const size_t bytes = bytes_.load(std::memory_order_relaxed), at = (size_t)(uint32_t)v * kPiece;
      if ((uint32_t)v == kClosed || at >= bytes) return false;
      if (!next_.compare_exchange_weak(v, v + 1, std::memory_order_acq_rel)) continue;
      move(dst + at, src + at, bytes - at < kPiece ? bytes - at : kPiece, past_cache);
      done_.fetch_add(1, std::memory_order_release);
      return true;
    }
  }
  void work() {
    while (!stop_.load(std::memory_order_relaxed)) {
      const uint64_t seen = next_.load() >> 32;
      bool any = false;
      while (take_piece()) any = true;
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(any ? 200 : 0);
      while ((next_.load(std::memory_order_relaxed) >> 32) == seen && !stop_.load(std::memory_order_relaxed) &&
             std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      if ((next_.load() >> 32) != seen) continue;
      std::unique_lock<std::mutex> l(sleep_mutex_);
      asleep_.fetch_add(1);
      wake_.wait(l, [&] { return stop_.load() || (next_.load() >> 32) != seen; });
      asleep_.fetch_sub(1);
    }
  }
  std::vector<std::thread> workers_;
  std::mutex mutex_, sleep_mutex_;
  std::condition_variable wake_;
  std::atomic<int> asleep_{0};
  std::atomic<bool> stop_{false};
  std::atomic<char *> dst_{nullptr};
  std::atomic<const char *> src_{nullptr};
  std::atomic<size_t> bytes_{0};
  std::atomic<bool> past_cache_{false};
  std::atomic<uint64_t> next_{kClosed};   // job number << 32 | next piece to claim
  std::atomic<uint32_t> done_{0};
};

}  // namespace sbb

// Copies between pageable host memory and the device.
//
// What bounds them is the copy by the CPU: a pageable cudaMemcpy stages the data through the driver's pinned buffer with
// one thread (12 GB/s up, 21 GB/s down measured here, against some 55 GB/s of the link).  Here the pieces of a copy pass
// through four pinned slots, several threads copy between the slots and the caller's memory, and the link moves one slot
// while the next is filled or drained.
#include "sbb_host.cuh"

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace sbb {
namespace {

// ---- memcpy by several threads ------------------------------------------------------------------
// One job at a time, cut into pieces that the caller and the workers claim one by one: whoever is late, for a worker still
// waking up, finds nothing left.  Workers spin for a while after a job (a copy is a series of jobs) before they sleep.
class CopyThreads {
 public:
  static CopyThreads &get() {
    static CopyThreads t;
    return t;
  }
  void copy(void *dst, const void *src, size_t bytes) {
    if (bytes <= 2 * kPiece || workers_.empty() || !mutex_.try_lock()) {   // (busy with another thread's job)
      std::memcpy(dst, src, bytes);
      return;
    }
    const uint32_t pieces = (uint32_t)((bytes + kPiece - 1) / kPiece);
    const uint64_t generation = (next_.load(std::memory_order_relaxed) >> 32) + 1;
    dst_.store(static_cast<char *>(dst), std::memory_order_relaxed);
    src_.store(static_cast<const char *>(src), std::memory_order_relaxed);
    bytes_.store(bytes, std::memory_order_relaxed);
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
  static constexpr size_t kPiece = 128 << 10;
  static constexpr uint32_t kClosed = 0xFFFFFFFFu;
  CopyThreads() {
    unsigned n = std::thread::hardware_concurrency() / 2;
    if (n > 8) n = 8;
    for (unsigned k = 1; k < n; ++k) workers_.emplace_back([this] { work(); });
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
      const size_t bytes = bytes_.load(std::memory_order_relaxed), at = (size_t)(uint32_t)v * kPiece;
      if ((uint32_t)v == kClosed || at >= bytes) return false;
      if (!next_.compare_exchange_weak(v, v + 1, std::memory_order_acq_rel)) continue;
      std::memcpy(dst + at, src + at, bytes - at < kPiece ? bytes - at : kPiece);
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
  std::atomic<uint64_t> next_{kClosed};   // job number << 32 | next piece to claim
  std::atomic<uint32_t> done_{0};
};

constexpr int kSlots = 4, kKept = 4;      // contexts kept for later calls: 32 MB of pinned memory at most
constexpr size_t kSlotBytes = 2 << 20;
constexpr size_t kDirectBytes = 64 << 10;   // smaller copies go as the driver does them
constexpr size_t kPoolBytes = 256 << 20;    // device memory kept between calls

bool pinned(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// Pieces of a copy: about four for a small one, so that its parts overlap too, slots for a large one.
size_t piece_of(size_t bytes) {
  size_t n = (bytes / 4 + 0xFFFF) & ~(size_t)0xFFFF;
  if (n < (256u << 10)) n = 256u << 10;
  return n < kSlotBytes ? n : kSlotBytes;
}

}  // namespace

struct HostContext {
  int device = -1;
  cudaStream_t stream = nullptr;
  char *slot[kSlots] = {nullptr, nullptr, nullptr, nullptr};
  cudaEvent_t event[kSlots] = {nullptr, nullptr, nullptr, nullptr};
  int next = 0;
  cudaError_t create(int dev) {
    device = dev;
    cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    for (int k = 0; k < kSlots && e == cudaSuccess; ++k) {
      e = cudaEventCreateWithFlags(&event[k], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaHostAlloc(reinterpret_cast<void **>(&slot[k]), kSlotBytes, cudaHostAllocPortable);
    }
    return e;
  }
  ~HostContext() {
    for (int k = 0; k < kSlots; ++k) {
      if (slot[k]) cudaFreeHost(slot[k]);
      if (event[k]) cudaEventDestroy(event[k]);
    }
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {
std::mutex g_contexts_mutex;
std::vector<HostContext *> g_contexts;   // free ones, at most kKept; the process's end gives them back
}  // namespace

HostCall::HostCall() {
  int dev = 0;
  error_ = cudaGetDevice(&dev);
  if (error_ != cudaSuccess) return;
  {
    std::lock_guard<std::mutex> l(g_contexts_mutex);
    for (size_t k = 0; k < g_contexts.size(); ++k)
      if (g_contexts[k]->device == dev) {
        ctx_ = g_contexts[k];
        g_contexts.erase(g_contexts.begin() + (long)k);
        return;
      }
  }
  ctx_ = new HostContext();
  error_ = ctx_->create(dev);
}

HostCall::~HostCall() {
  if (ctx_ == nullptr) return;
  if (error_ == cudaSuccess) {
    std::lock_guard<std::mutex> l(g_contexts_mutex);
    if ((int)g_contexts.size() < kKept) {
      g_contexts.push_back(ctx_);
      return;
    }
  }
  for (int k = 0; k < kSlots; ++k)
    if (ctx_->event[k]) cudaEventSynchronize(ctx_->event[k]);
  delete ctx_;
}

cudaStream_t HostCall::stream() const { return ctx_->stream; }

cudaError_t HostCall::upload(void *dev, const void *host, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  if (bytes <= kDirectBytes || pinned(host)) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
  const size_t piece = piece_of(bytes);
  for (size_t at = 0; at < bytes; at += piece) {
    const size_t n = bytes - at < piece ? bytes - at : piece;
    const int k = ctx_->next;
    ctx_->next = (k + 1) % kSlots;
    cudaError_t e = cudaEventSynchronize(ctx_->event[k]);   // the slot's last copy has left it
    if (e != cudaSuccess) return e;
    CopyThreads::get().copy(ctx_->slot[k], static_cast<const char *>(host) + at, n);
    e = cudaMemcpyAsync(static_cast<char *>(dev) + at, ctx_->slot[k], n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaEventRecord(ctx_->event[k], st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t HostCall::download(void *host, const void *dev, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return cudaStreamSynchronize(st);
  if (bytes <= kDirectBytes || pinned(host)) {
    cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
    return e != cudaSuccess ? e : cudaStreamSynchronize(st);
  }
  const size_t piece = piece_of(bytes), pieces = (bytes + piece - 1) / piece;
  const int first = ctx_->next;
  auto length = [&](size_t p) { return bytes - p * piece < piece ? bytes - p * piece : piece; };
  auto request = [&](size_t p) -> cudaError_t {   // (a slot is asked for again only when its piece has been copied out)
    const int k = (int)((first + p) % kSlots);
    cudaError_t e = cudaSuccess;
    if (p < (size_t)kSlots) e = cudaEventSynchronize(ctx_->event[k]);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(ctx_->slot[k], static_cast<const char *>(dev) + p * piece, length(p), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(ctx_->event[k], st);
    return e;
  };
  for (size_t p = 0; p < pieces && p < (size_t)kSlots; ++p) {
    const cudaError_t e = request(p);
    if (e != cudaSuccess) return e;
  }
  for (size_t p = 0; p < pieces; ++p) {
    const int k = (int)((first + p) % kSlots);
    cudaError_t e = cudaEventSynchronize(ctx_->event[k]);
    if (e != cudaSuccess) return e;
    CopyThreads::get().copy(static_cast<char *>(host) + p * piece, ctx_->slot[k], length(p));
    if (p + kSlots < pieces && (e = request(p + kSlots)) != cudaSuccess) return e;
  }
  ctx_->next = (int)((first + pieces) % kSlots);
  return cudaSuccess;
}

namespace {
// A pool of our own, so that its bound touches nobody else's allocations.
cudaError_t pool_of(int dev, cudaMemPool_t *out) {
  static std::mutex mutex;
  static cudaMemPool_t pools[64];
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> l(mutex);
  if (pools[dev] == nullptr) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    uint64_t keep = kPoolBytes;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) return e;
    pools[dev] = p;
  }
  *out = pools[dev];
  return cudaSuccess;
}
}  // namespace

cudaError_t HostCall::allocate(void **dev, size_t bytes, cudaStream_t st) {
  int d = 0;
  cudaMemPool_t pool;
  cudaError_t e = cudaGetDevice(&d);
  if (e == cudaSuccess) e = pool_of(d, &pool);
  return e == cudaSuccess ? cudaMallocFromPoolAsync(dev, bytes, pool, st) : e;
}
void HostCall::free(void *dev, cudaStream_t st) {
  if (dev) cudaFreeAsync(dev, st);
}

}  // namespace sbb

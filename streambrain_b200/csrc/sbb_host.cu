// Copies between pageable host memory and the device.
//
// A pageable cudaMemcpy stages the data through the driver's pinned buffer with one thread (12 GB/s up, 21 GB/s down measured
// here, against some 50 GB/s of the link, which moves as much in both directions at once).  Here the pieces of a copy pass
// through pinned slots, several threads copy between a slot and the caller's memory (50 to 150 GB/s; one thread 12), and the link
// moves one slot while the next is filled or drained.  A copy over the link costs 6 us whatever its size: small buffers that
// lie behind one another on the device travel together.
#include "sbb_host.cuh"

#include <cstdint>
#include <mutex>
#include <new>

#include "sbb_copy_threads.h"

namespace sbb {
namespace {

constexpr int kUp = 2, kDown = 4, kKept = 4;   // slots; contexts kept for later calls: 96 MB of pinned memory at most
constexpr int kRanges = 8;                // host buffers that share a copy
constexpr size_t kSlotBytes = HostCall::kSlot;
constexpr size_t kDirectBytes = 64 << 10;   // smaller copies of a single buffer go as the driver does them
constexpr size_t kPoolBytes = 256 << 20;    // device memory kept between calls

bool pinned(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// Pieces of a copy: two or three for a small one, so that its parts overlap too, half slots for a large one.
size_t piece_of(size_t bytes) {
  size_t n = (bytes / 3 + 0xFFFF) & ~(size_t)0xFFFF;
  if (n < (512u << 10)) n = 512u << 10;
  return n < kSlotBytes / 2 ? n : kSlotBytes / 2;
}

}  // namespace

struct HostContext {
  int device = -1;
  cudaStream_t stream = nullptr, out = nullptr;
  cudaEvent_t mark = nullptr;
  struct Slot {
    char *mem = nullptr;
    cudaEvent_t event = nullptr;   // its last copy over the link is through
  };
  Slot up[kUp], down[kDown];
  // what a down slot holds for the host: the bytes [at, at + bytes) of the ranges' device space
  struct Pending {
    HostCall::Range range[kRanges];
    int ranges = 0;
    size_t at = 0, bytes = 0;
  };
  Pending pending[kDown];
  int next_up = 0, next_down = 0;
  cudaError_t create(int dev) {
    device = dev;
    cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&out, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&mark, cudaEventDisableTiming);
    for (int k = 0; k < kUp + kDown && e == cudaSuccess; ++k) {
      Slot &s = k < kUp ? up[k] : down[k - kUp];
      e = cudaEventCreateWithFlags(&s.event, cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaHostAlloc(reinterpret_cast<void **>(&s.mem), kSlotBytes, cudaHostAllocPortable);
    }
    return e;
  }
  ~HostContext() {
    for (int k = 0; k < kUp + kDown; ++k) {
      Slot &s = k < kUp ? up[k] : down[k - kUp];
      if (s.mem) cudaFreeHost(s.mem);
      if (s.event) cudaEventDestroy(s.event);
    }
    if (mark) cudaEventDestroy(mark);
    if (out) cudaStreamDestroy(out);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {
std::mutex g_contexts_mutex;
HostContext *g_contexts[kKept];   // free ones; the process's end gives them back
int g_free_contexts = 0;
}  // namespace

HostCall::HostCall() {
  int dev = 0;
  error_ = cudaGetDevice(&dev);
  if (error_ != cudaSuccess) return;
  {
    std::lock_guard<std::mutex> l(g_contexts_mutex);
    for (int k = 0; k < g_free_contexts; ++k)
      if (g_contexts[k]->device == dev) {
        ctx_ = g_contexts[k];
        g_contexts[k] = g_contexts[--g_free_contexts];
        return;
      }
  }
  ctx_ = new (std::nothrow) HostContext();
  error_ = ctx_ != nullptr ? ctx_->create(dev) : cudaErrorMemoryAllocation;
}

HostCall::~HostCall() {
  if (ctx_ == nullptr) return;
  for (int k = 0; k < kDown; ++k) ctx_->pending[k].bytes = 0;   // (a call that failed: nobody waits for these)
  if (error_ == cudaSuccess) {
    std::lock_guard<std::mutex> l(g_contexts_mutex);
    if (g_free_contexts < kKept) {
      g_contexts[g_free_contexts++] = ctx_;
      return;
    }
  }
  for (int k = 0; k < kUp + kDown; ++k) {
    const cudaEvent_t event = k < kUp ? ctx_->up[k].event : ctx_->down[k - kUp].event;
    if (event) cudaEventSynchronize(event);
  }
  delete ctx_;
}

cudaStream_t HostCall::stream() const { return ctx_->stream; }
cudaStream_t HostCall::stream_out() const { return ctx_->out; }
cudaError_t HostCall::out_after(cudaStream_t st) {
  const cudaError_t e = cudaEventRecord(ctx_->mark, st);
  return e == cudaSuccess ? cudaStreamWaitEvent(ctx_->out, ctx_->mark, 0) : e;
}

namespace {
// Copies the bytes [at, at + bytes) of the ranges' device space between the slot and the host.
void exchange(const HostCall::Range *range, int ranges, size_t at, size_t bytes, char *slot, bool to_host) {
  for (int r = 0; r < ranges; ++r) {
    const size_t lo = range[r].offset > at ? range[r].offset : at;
    const size_t end = range[r].offset + range[r].bytes, hi = end < at + bytes ? end : at + bytes;
    if (lo >= hi) continue;
    char *host = static_cast<char *>(range[r].host) + (lo - range[r].offset), *piece = slot + (lo - at);
    if (to_host) CopyThreads::get().copy(host, piece, hi - lo, true);
    else CopyThreads::get().copy(piece, host, hi - lo);
  }
}
// How many of the ranges, from the first on, go through the slots together: up to the next page-locked one, which the link
// reaches by itself (0: that is the first).
int staged(const HostCall::Range *range, int ranges) {
  int n = 0;
  while (n < ranges && !(range[n].bytes > kDirectBytes && pinned(range[n].host))) ++n;
  return n;
}
}  // namespace

cudaError_t HostCall::upload(void *dev, const void *host, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  if (bytes <= kDirectBytes) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
  const Range r{const_cast<void *>(host), 0, bytes};
  return upload(dev, &r, 1, st);
}

cudaError_t HostCall::upload(void *dev, const Range *range, int ranges, cudaStream_t st, size_t most) {
  cudaError_t e = cudaSuccess;
  for (int r = 0; r < ranges && e == cudaSuccess;) {
    const int n = staged(range + r, ranges - r);
    if (n == 0) {
      e = cudaMemcpyAsync(static_cast<char *>(dev) + range[r].offset, range[r].host, range[r].bytes, cudaMemcpyHostToDevice, st);
      ++r;
      continue;
    }
    const size_t begin = range[r].offset, end = range[r + n - 1].offset + range[r + n - 1].bytes, piece = most != 0 ? most : piece_of(end - begin);
    for (size_t at = begin; at < end && e == cudaSuccess; at += piece) {
      const size_t bytes = end - at < piece ? end - at : piece;
      HostContext::Slot &slot = ctx_->up[ctx_->next_up];
      ctx_->next_up = (ctx_->next_up + 1) % kUp;
      e = cudaEventSynchronize(slot.event);   // the slot's last copy has left it
      if (e != cudaSuccess) break;
      exchange(range + r, n, at, bytes, slot.mem, false);
      e = cudaMemcpyAsync(static_cast<char *>(dev) + at, slot.mem, bytes, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaEventRecord(slot.event, st);
    }
    r += n;
  }
  return e;
}

// What the slot holds reaches the host.
cudaError_t HostCall::drain(int k) {
  HostContext::Pending &p = ctx_->pending[k];
  if (p.bytes == 0) return cudaSuccess;
  const cudaError_t e = cudaEventSynchronize(ctx_->down[k].event);
  if (e == cudaSuccess) exchange(p.range, p.ranges, p.at, p.bytes, ctx_->down[k].mem, true);
  p.bytes = 0;
  return e;
}

cudaError_t HostCall::request(void *host, const void *dev, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  const Range r{host, 0, bytes};
  return request(&r, 1, dev, st);
}

cudaError_t HostCall::request(const Range *range, int ranges, const void *dev, cudaStream_t st, size_t most) {
  cudaError_t e = cudaSuccess;
  for (int r = 0; r < ranges && e == cudaSuccess;) {
    const int n = staged(range + r, ranges - r < kRanges ? ranges - r : kRanges);
    if (n == 0) {
      e = cudaMemcpyAsync(range[r].host, static_cast<const char *>(dev) + range[r].offset, range[r].bytes, cudaMemcpyDeviceToHost, st);
      ++r;
      continue;
    }
    const size_t begin = range[r].offset, end = range[r + n - 1].offset + range[r + n - 1].bytes, piece = most != 0 ? most : piece_of(end - begin);
    for (size_t at = begin; at < end && e == cudaSuccess; at += piece) {
      const size_t bytes = end - at < piece ? end - at : piece;
      const int k = ctx_->next_down;
      ctx_->next_down = (k + 1) % kDown;
      e = drain(k);
      if (e == cudaSuccess) e = cudaEventSynchronize(ctx_->down[k].event);   // (a failed call's copy)
      if (e == cudaSuccess) e = cudaMemcpyAsync(ctx_->down[k].mem, static_cast<const char *>(dev) + at, bytes, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(ctx_->down[k].event, st);
      if (e != cudaSuccess) break;
      HostContext::Pending &p = ctx_->pending[k];
      for (int q = 0; q < n; ++q) p.range[q] = range[r + q];
      p.ranges = n;
      p.at = at;
      p.bytes = bytes;
    }
    r += n;
  }
  return e;
}

cudaError_t HostCall::finish(cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < kDown && e == cudaSuccess; ++q) e = drain((ctx_->next_down + q) % kDown);   // in the order of the requests
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
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

// Copies between pageable host memory and the device.
//
// What bounds them is the copy by the CPU: a pageable cudaMemcpy stages the data through the driver's pinned buffer with
// one thread (12 GB/s up, 21 GB/s down measured here, against some 55 GB/s of the link).  Here the pieces of a copy pass
// through four pinned slots, and the link moves one slot while the next is filled or drained; pieces of more than 256 KB,
// that is copies of more than 1 MB, are copied between the slots and the caller's memory by several threads.
#include "sbb_host.cuh"

#include <cstdint>
#include <mutex>
#include <new>

#include "sbb_copy_threads.h"

namespace sbb {
namespace {

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
  if (error_ == cudaSuccess) {
    std::lock_guard<std::mutex> l(g_contexts_mutex);
    if (g_free_contexts < kKept) {
      g_contexts[g_free_contexts++] = ctx_;
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

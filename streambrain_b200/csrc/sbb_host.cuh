// Copies between pageable host memory and the device, and the device memory of one host-buffer call.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace sbb {

// What a call on host buffers works with on the current device: a stream of its own and pinned slots its copies pass
// through.  Taken from a process-wide set; the destructor gives it back.  Safe with several threads.
struct HostContext;
class HostCall {
 public:
  HostCall();
  ~HostCall();
  HostCall(const HostCall &) = delete;
  HostCall &operator=(const HostCall &) = delete;
  cudaError_t error() const { return error_; }
  cudaStream_t stream() const;
  cudaStream_t stream_out() const;   // a second one, for copies to the host beside those from it
  cudaError_t out_after(cudaStream_t st);   // what is queued on stream_out() from here on waits for what is queued on `st` now
  // Queued on `st`; the host buffer has been read when the call returns, or (page-locked memory) when `st` gets there.
  cudaError_t upload(void *dev, const void *host, size_t bytes, cudaStream_t st);
  static constexpr size_t kSlot = 4 << 20;   // bytes of a pinned slot: the longest piece of a copy
  // The same for several host buffers that lie behind one another on the device, small ones in one copy: `range` in
  // ascending order of `offset`, which counts from `dev`; what lies between them is overwritten.
  // `piece` (up to kSlot): into pieces of this many bytes instead of those that suit a copy by itself.
  struct Range {
    void *host;
    size_t offset, bytes;
  };
  cudaError_t upload(void *dev, const Range *range, int ranges, cudaStream_t st, size_t piece = 0);
  // Queued on `st`; the host buffers are complete when finish() returns, which waits for all that has been requested.
  cudaError_t request(void *host, const void *dev, size_t bytes, cudaStream_t st);
  cudaError_t request(const Range *range, int ranges, const void *dev, cudaStream_t st, size_t piece = 0);
  cudaError_t finish(cudaStream_t st);
  // Waits for `st`; the host buffer is complete when the call returns.
  cudaError_t download(void *host, const void *dev, size_t bytes, cudaStream_t st) {
    const cudaError_t e = request(host, dev, bytes, st);
    return e == cudaSuccess ? finish(st) : e;
  }
  // Device memory, ordered on `st` (from a pool that keeps freed memory for the next call, up to a bound).
  static cudaError_t allocate(void **dev, size_t bytes, cudaStream_t st);
  static void free(void *dev, cudaStream_t st);

 private:
  cudaError_t drain(int slot);
  HostContext *ctx_ = nullptr;
  cudaError_t error_ = cudaSuccess;
};

}  // namespace sbb

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
  // Queued on `st`; the host buffer has been read when the call returns, or (page-locked memory) when `st` gets there.
  cudaError_t upload(void *dev, const void *host, size_t bytes, cudaStream_t st);
  // Waits for `st`; the host buffer is complete when the call returns.
  cudaError_t download(void *host, const void *dev, size_t bytes, cudaStream_t st);
  // Device memory, ordered on `st` (from a pool that keeps freed memory for the next call, up to a bound).
  static cudaError_t allocate(void **dev, size_t bytes, cudaStream_t st);
  static void free(void *dev, cudaStream_t st);

 private:
  HostContext *ctx_ = nullptr;
  cudaError_t error_ = cudaSuccess;
};

}  // namespace sbb

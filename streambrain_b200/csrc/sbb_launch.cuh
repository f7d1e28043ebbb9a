// Launches that begin while the kernel before them in the stream drains (programmatic stream serialization).
#pragma once
#include <cuda_runtime.h>

namespace sbb {

// First statement of a kernel that launch_next starts, ahead of every access to global memory: waits until the kernels
// before it in the stream have ended and what they wrote is visible, then lets the next kernel's blocks take the places that
// this kernel's leave.  Every kernel of a chain waits, so each has all its predecessors behind it.
// Two kernels wait later, only ahead of what the kernel directly before them in the stream writes: the trace updates of
// sbb_tc_trace.cu and sbb_f64_mma.cuh, whose products and old traces do not depend on the column vectors formed there.
// All that is older has ended before their blocks may start, because the kernel before let them start only after its own
// wait.  Their launchers' declarations say what that kernel may not write.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A training step is five kernels of 3 to 30 us; starting each only when the one before had ended cost 1.1 to 2.5 us a
// launch.  1001 x 481 at batch 97: 49 -> 40 us a step; 1568 x 3000 at 128: 74 -> 68; a fit of 5000 samples: 6.7 -> 5.4 ms.
template <class... P, class... A>
inline cudaError_t launch_next(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

// The same in clusters of blocks.
template <class... P, class... A>
inline cudaError_t launch_clusters(void (*kernel)(P...), dim3 grid, dim3 cluster, unsigned threads, size_t smem, cudaStream_t st,
                                   A... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster.x;
  attr[1].val.clusterDim.y = cluster.y;
  attr[1].val.clusterDim.z = cluster.z;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

}  // namespace sbb

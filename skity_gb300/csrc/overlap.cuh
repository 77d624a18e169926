// Overlapped launches (programmatic dependent launch): a kernel may start when
// every CTA of the kernel before it on the stream has started and allowed it,
// and waits inside for that kernel's work to be complete and visible.
#pragma once
#include <cuda_runtime.h>

namespace skc {

// Lets the next overlapped launch start once every CTA of this one runs.
__device__ __forceinline__ void AllowNextLaunch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Waits for the kernel before to be complete (returns at once in a launch
// that overlaps nothing).  A kernel all of whose threads call this completes
// after everything before it on the stream.
__device__ __forceinline__ void WaitLaunchBefore() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// overlap: the kernel may start before the one before it is complete.
template <typename... Args>
inline void LaunchOverlapped(void (*kernel)(Args...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, bool overlap, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace skc

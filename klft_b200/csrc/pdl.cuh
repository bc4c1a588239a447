// pdl.cuh -- programmatic dependent launch: a kernel launched as a dependent of the
// one before it in its stream is brought onto the device while that one still
// runs, and waits there; chains of short kernels lose the time between the end of
// one and the start of the next.
//
// A kernel launched this way calls grid_dependency_wait() before it reads or writes
// any memory another kernel touches, and at least one of its threads calls it, so
// that "the kernel before has ended" includes all kernels before that.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace klft {

__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// dependent: the operation before in the stream is a kernel (else an ordinary launch).
// A launch that is refused does not leave its error behind for the next call to report.
template <typename... KArgs, typename... Args>
cudaError_t launch_after(bool dependent, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                         Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = dependent ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

}  // namespace klft

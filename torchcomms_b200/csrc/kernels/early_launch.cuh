// Programmatic dependent launch: a kernel whose blocks start while the kernel in front of it on the stream still runs.
//
// Between two kernels of a stream lie some 2 us (the first one's last blocks, its flush, the next one's launch) and each
// kernel then sets up barriers, tensor memory and descriptors before it touches data. A kernel launched with
// launch_early() does that part early; grid_wait() holds it until every grid in front of it is complete and its writes
// are visible. The rules that keep this as safe as an ordinary launch:
//   - nothing is read from or written to global memory before grid_wait(), in any thread;
//   - every block passes grid_wait(), so that a kernel is complete only after the ones in front of it are;
//   - what a kernel reads may have been written while its blocks were already resident, so it is read with ordinary
//     loads or TMA, never through the read-only path (no __ldg, no const __restrict__ pointers).
// grid_release() lets the next kernel's blocks take the room that this one leaves; they wait at their own grid_wait().
#pragma once

#include <cuda_runtime.h>

namespace b200c {

#ifdef __CUDACC__

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_early(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

#endif // __CUDACC__

} // namespace b200c

// Launches of a plan's kernel sequences with programmatic dependent launch: a kernel's CTAs are
// set up as the last ones of the kernel before leave, and wait in grid_wait() for its end, so the
// next launch overlaps the drain and the memory flush of the last.  An explicit iteration is 12
// dependent launches of 2 to 14 us: 60 iterations of three 128x48 cases in FP64 take 8.3 ms with
// plain launches and 7.0 with these, 40 of 32 256x64 cases in FP32 13.2 and 12.2.  A Newton step's
// graph takes the same time either way.  Letting the next kernel in earlier, by
// griddepcontrol.launch_dependents at the start, made the explicit iterations slower (8.9 ms).
#pragma once
#include <cuda_runtime.h>

namespace a2d {

// First statement of every kernel that launch() starts: before it the kernel ahead in the stream
// may still be running, after it that one has ended and all that it wrote is visible.  No path may
// leave such a kernel without it: a kernel that ended early would let its successor, which waits
// for this one alone, run beside its predecessor.
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

inline cudaLaunchAttribute dependent_launch() {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  return at;
}

// k<<<grid, block, smem, s>>>(args...); errors are left for cudaGetLastError, as there
template <typename... P, typename... A>
inline void launch(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at = dependent_launch();
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

}  // namespace a2d

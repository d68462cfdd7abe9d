// Programmatic dependent launch: a kernel's blocks may become resident, and set up, while the kernel before it in the stream ends.
// Between two kernels of a few us that is 1 to 1.5 us, and the launch itself takes the host 2.2 us instead of 2.6: the linear layer
// of 1992 x 4104 x 1032 81.7 -> 78.5 us, of 512 x 512 x 1536 26.4 -> 24.8, a two-layer model of width 512 481 -> 453; calls of
// several hundred us stay as they are.  Kernels of a row exchange, which wait for other GPUs, are launched plainly.
#pragma once
#include <cuda_runtime.h>

namespace msb {

// Wait until the grids before this one in the stream are complete and their writes visible / let the next grid start once every
// block of this one has come here or left.  In a grid that was launched plainly the wait does nothing, but the trigger counts:
// a kernel of a row exchange does not come to it, or what follows would take SMs while it waits for other GPUs.  Every block of a
// grid launched with launch_dependent() waits, before it touches memory that an earlier grid may use: then what follows this grid
// follows those too.
// Such a kernel runs while its inputs are still being written, so none of its pointers is __restrict__: a const one would let
// the compiler load through the non-coherent path, or take a load for invariant and move it over the wait.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  // a refusal is this call's answer, and not also that of the next one that asks for the last error
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

}  // namespace msb

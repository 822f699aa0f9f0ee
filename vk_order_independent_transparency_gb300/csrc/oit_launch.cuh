// Launches of the frame's kernels with programmatic stream serialization: a
// frame is a chain of ten short kernels, and with it the next kernel's launch
// is under way before the one before it has drained. Every kernel launched
// this way calls frame_order() before it touches memory: it waits until all
// work before it has completed and is visible. It then reads global memory with
// ordinary loads (or volatile ones with a cache operator) through plain
// pointers. __ldg, and __restrict__ on its parameters, tell the compiler that
// nothing else writes that memory while the kernel runs, but the kernel may
// have begun before its predecessor wrote it: such a load need not stay behind
// the wait, nor see what the wait makes visible. Only the constant tables of
// oit_device.cuh are read through __ldg.
// Frames of single calls, without and with it: Spinlock 64x40 51 -> 28 us,
// 800x512 242 -> 205 us, WBOIT 641x359 116 -> 93 us, Simple 1283x717 4x MSAA 350
// -> 302 us (a replayed graph gains nothing). Letting the next kernel be placed
// as soon as all blocks run (griddepcontrol.launch_dependents) measured up to
// 5% slower than at their end: its waiting blocks hold registers and shared
// memory.
#pragma once

#include <cuda_runtime.h>

namespace oitd {

__device__ __forceinline__ void frame_order() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_in_frame(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace oitd

// Launches whose set-up overlaps the kernel before them on the stream, and warps
// that take places from a counter together.
//
// A tree build is a chain of small kernels, 4 to 9 us each, and as much again of
// their time lies between them; a frame's stages are such a chain too. A kernel
// launched with launch_after may be set up while the kernel before it still runs; it
// begins with wait_previous(), which returns when that kernel has completed and its
// writes are visible. Every block of such a kernel calls it first, before any return,
// and the kernel reads nothing through the non-coherent path (__ldg, const
// __restrict__) that an earlier kernel of the chain writes.
//
// after_previous() also lets the blocks of the next kernel be placed right away, to
// wait there: for the builds' kernels, which don't fill the chip (a 20,480-triangle
// reference-rule build of 9 levels 642 -> 542 us). The stages fill it, and blocks
// that wait would hold the places of the other frames in flight: four frames of
// 641x360 948 us with plain launches, 826 with wait_previous(), 1,072 with
// after_previous().
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ct {

__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
  wait_previous();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// chained false: an ordinary launch. A kernel whose stream waits for an event of another
// stream right before it is launched so (ray generation, a shade that joins a connect).
template <class... P, class... A>
inline cudaError_t launch_after_if(bool chained, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                                   cudaStream_t s, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = a;
  c.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                                A... args) {
  return launch_after_if(true, kernel, grid, block, smem, s, args...);
}

// Places for a warp's threads that want `want` units each from a counter, with one
// atomic for the warp.
__device__ __forceinline__ uint32_t warp_alloc(uint32_t* counter, uint32_t want) {
  const int lane = threadIdx.x & 31;
  uint32_t inc = want;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += y;
  }
  uint32_t base = 0;
  if (lane == 31 && inc) base = atomicAdd(counter, inc);
  return __shfl_sync(0xffffffffu, base, 31) + inc - want;
}

}  // namespace ct

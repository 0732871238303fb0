// Launches whose set-up overlaps the kernel before them on the stream, and warps
// that take places from a counter together.
//
// A tree build is a chain of small kernels: for 20,480 triangles five kernels of 4
// to 9 us a level, and as much again of their time between them. A kernel launched
// with launch_after may be set up, and its blocks placed, while the kernel before it
// still runs; it begins with after_previous(), which waits until that kernel has
// completed and its writes are visible, and then lets the next one be set up.
// Every block of such a kernel calls it first, before any return, and the kernel
// reads nothing through the non-coherent path (const __restrict__) that an earlier
// kernel of the chain writes. With plain launches a 20,480-triangle reference-rule
// build (9 levels) took 642 us, so 542.
#pragma once
#include <cuda_runtime.h>

namespace ct {

__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                                A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = a;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
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

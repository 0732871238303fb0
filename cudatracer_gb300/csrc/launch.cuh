// Launches whose set-up overlaps the kernel before them on the stream.
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

}  // namespace ct

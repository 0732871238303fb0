// Allocation-free render path: frames for which the library allocates nothing.
//
// Who needs it: a host application that owns all device memory itself, or
// whose render thread must never enter the CUDA allocator (cudaMalloc and
// cudaFree can synchronise the device and stall the frame). Such a caller
// creates its scene and BVH once at load time, then renders every frame
// through ct_render_accumulate_noalloc into an accumulation buffer it owns.
//
// Limits and sharing:
//   * at most kNoAllocMaxPixels paths per frame (width * height <= 65,536,
//     e.g. 256 x 256). Every such frame is the one kernel of small frames
//     (launch_path), which keeps a path in a thread's registers and needs no
//     queues: the stages took 540 us at 160x120, the kernel
//     takes 182 (64x48: 460 and 107, 256x256: 610 and 218);
//   * the kernel counts its rays in a few static words that nobody reads;
//   * the first call on each device looks up the words' device address
//     with cudaGetSymbolAddress; make that first call before any stream
//     capture begins. The address is kept for the life of the process and
//     belongs to the device's context as it was then: after a cudaDeviceReset
//     of that device it is stale, so the entry point must not be used on a
//     device this process has reset since its first call there.
#include <mutex>

#include "ct_internal.h"

namespace ct {

constexpr uint32_t kNoAllocMaxPixels = 65536;
static __device__ unsigned long long g_noalloc_stats[8];

namespace {
std::mutex g_mu;
void* g_addr[256] = {};  // per device ordinal, looked up once
}  // namespace

uint32_t noalloc_max_pixels() { return kNoAllocMaxPixels; }

// Looks the address up once per device (with that device current).
cudaError_t noalloc_stats(int device, unsigned long long** out) {
  if (device < 0 || device >= 256) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(g_mu);
  if (!g_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_stats);
    if (e != cudaSuccess) return e;
    g_addr[device] = p;
  }
  *out = (unsigned long long*)g_addr[device];
  return cudaSuccess;
}

cudaError_t noalloc_render(int device, const DevScene& sc, const DevBVH& bvh, const FrameConst& f, int max_depth,
                           int exact_math, float4* accum, uint32_t* err, cudaStream_t s) {
  DevQueues q{};
  cudaError_t e = noalloc_stats(device, &q.stats);
  if (e != cudaSuccess) return e;
  q.accum = accum;
  q.error = err;
  q.capacity = f.width * f.height;
  return launch_path(sc, bvh, q, f, max_depth, math_exact_shading(exact_math), math_fast_traversal(exact_math), s);
}

}  // namespace ct

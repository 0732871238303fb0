// Device BVH builder: the reference's binned SAH (src/BVH/BVHNode.cu:121-190)
// and MergeNodes collapse (src/BVH/MBVHNode.cu:27-61, 226-277) run on the GPU.
//
// The split rule is the host builder's, evaluated with the same IEEE
// operations (no contraction: __fadd_rn/__fmul_rn/__fdiv_rn): ten planes per
// axis at min + len*i/11, a primitive's interval = the number of planes its
// centroid is not <= to, cost = area(left)*nl + area(right)*nr, the first
// lowest cost in axis-outer/plane-inner order, a leaf when the parent's cost
// is lower, when fewer than 4 primitives remain, or at binary depth 62. Bin
// boxes are unions (exact min/max), so every node box, count and primitive
// range equals the host build's: the quad tree comes out bit-identical, with
// the primitives of each leaf in another order (both partitions here are
// stable; the reference's swap partition is not).
//
// Phases:
//   prep      per-primitive padded bounds (triangle::getBounds) and the root box
//   levels    nodes with more than mid_size(n) primitives, level by level: chunks of
//             primitives bin into shared memory and flush to the node's global
//             bins; one warp per node picks the split; a bit per primitive and
//             chunk counts give a stable partition into the other level's buffer
//   mid       one block splits each node down to ranges of <= kWarpMax in shared
//             memory
//   small     one warp splits the subtree of each node of <= kWarpMax primitives
//             down to ranges of <= kLeafTask, bins and partition in shared memory
//   leaf      one thread builds the whole subtree of each such range
//   collapse  quad nodes are the inner binary nodes at even depth; subtree
//             quad counts bottom-up (arrival counters), each quad node's
//             pre-order index from its ancestors' left-sibling counts, then
//             every quad node written in place, as MergeNodes numbers them
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <memory>
#include <new>

#include "bvh_build.h"
#include "ct_internal.h"
#include "launch.cuh"

namespace ct {
namespace {

constexpr int kPlanes = 10;
constexpr int kIntervals = kPlanes + 1;
constexpr int kBinFields = 7;  // count, min key x/y/z, max key x/y/z
constexpr int kBinWords = 3 * kIntervals * kBinFields;
constexpr uint32_t kWarpMax = 128;  // nodes up to this size are built by one warp
// Nodes up to this size are split by one block down to those (64 KB of shared memory
// leave three blocks of 2,048 on an SM and six of 1,024). Terrains with 2,048 and with
// 1,024, ms: 486,000 triangles 1.22 and 1.22, 864,000 1.74 and 1.69, 1.5 M 2.53 and 2.48.
inline uint32_t mid_size(uint32_t n) { return n > 400000 ? 1024 : 2048; }
// Builds of at most this many triangles leave an SM about one such block, which has 512
// threads then instead of 256. Terrains with 256 and with 512 threads, us: 122,000
// triangles 836 and 820, 231,000 977 and 960, 302,000 1,029 and 1,046, 602,000 1,406 and
// 1,508.
constexpr uint32_t kFewMid = 250000;
constexpr uint32_t kLeafTask = 16;  // subtrees up to this size are built by one thread
// Primitives per block of the level kernels: the fewest, as a power of two from
// 256, that leave no more blocks than about one wave holds (8 blocks of 256 threads
// on each SM). A 20,480-triangle build has 80 blocks of one pass over
// their threads rather than 10 of eight (k_bin 18 -> 8 us a level); above 1.2 M
// triangles the 2,048 of one wave stay (fewer bin flushes).
inline uint32_t chunk_size(uint32_t n) {
  uint32_t c = 256;
  while (c < 2048 && n / c > (uint32_t)sm_count() * 8) c *= 2;
  return c;
}
constexpr int32_t kMaxSplitDepth = 61;
constexpr int kSmallStack = 64;
constexpr int kSmallWarps = 8;

enum : uint32_t { kErrDegenerate = 1, kErrArena = 2, kErrStack = 4, kErrPartition = 8 };
enum Counter : int {
  kArenaCount = 0,
  kSmallCount = 1,
  kChunks = 2,       // 2 words: chunks of the even and of the odd level
  kTasks = kChunks,  // ranges for k_leaf, once the levels are done
  kError = 4,
  kMaxLeaf = 5,
  kQuadDepth = 6,
  kMid = 7,          // nodes for k_mid
  kRootKeys = 8,     // 6 words: min x/y/z, max x/y/z
  kLarge = 14,       // 2 words: large nodes of the even and of the odd level
  kCounterWords = 16
};

struct __align__(16) BNode {
  float mn[3];
  int32_t first;
  float mx[3];
  int32_t count;
  int32_t left;    // -1 for a leaf, else the left child (right = left + 1)
  int32_t parent;  // -1 at the root
  int32_t depth;
  uint32_t qcount;  // quad nodes in the subtree (collapse phase)
};
static_assert(sizeof(BNode) == 48, "BNode");

// A primitive's box: 32 bytes, one load and one sector wherever it lies (the
// kernels read primitives in the order of the ranges they make).
struct __align__(32) PrimBox {
  float4 lo, hi;
};
__device__ __forceinline__ PrimBox prim_box(const PrimBox* b) {
  PrimBox v;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v.lo.x), "=f"(v.lo.y), "=f"(v.lo.z), "=f"(v.lo.w), "=f"(v.hi.x), "=f"(v.hi.y), "=f"(v.hi.z), "=f"(v.hi.w)
      : "l"(b));
  return v;
}

struct Chunk {
  int32_t slot;
  uint32_t begin, end;
};
struct Split {
  int32_t axis;  // -1: the node stays a leaf
  float coord;
  uint32_t lc;
  uint32_t chunk0;
  uint32_t queued;  // bit 0, 1: the left, right child is split on the next level
};

// Carving of the scratch block for n primitives.
struct Layout {
  size_t box, prims, tmp, arena, arrive, qidx, large0, large1, mid, small, chunks, chunk_left, split, bins,
      counters, total;
  uint32_t chunk, cap, mid_most, max_large, max_mid, max_chunks, max_small;
  explicit Layout(uint32_t n) {
    cap = 2 * n + 2;
    mid_most = mid_size(n);
    max_large = n / (mid_most + 1) + 2;
    max_mid = n / (kWarpMax + 1) + 2;
    chunk = chunk_size(n);
    max_chunks = n / chunk + max_large + 2;
    max_small = n / 4 + 2;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += (bytes + 255) & ~(size_t)255;
      return at;
    };
    box = take(sizeof(PrimBox) * (size_t)n);
    prims = take(4 * (size_t)n);
    tmp = take(4 * (size_t)n);
    arena = take(sizeof(BNode) * (size_t)cap);
    arrive = take(4 * (size_t)cap);
    qidx = take(4 * (size_t)cap);
    large0 = take(4 * (size_t)max_large);
    large1 = take(4 * (size_t)max_large);
    mid = take(4 * (size_t)max_mid);
    small = take(4 * (size_t)max_small);
    chunks = take(sizeof(Chunk) * (size_t)max_chunks);
    chunk_left = take(4 * (size_t)max_chunks);
    split = take(sizeof(Split) * (size_t)max_large);
    bins = take(4 * (size_t)kBinWords * max_large);
    counters = take(4 * kCounterWords);
    total = o;
  }
};

template <typename T>
T* at(void* base, size_t off) {
  return reinterpret_cast<T*>(static_cast<char*>(base) + off);
}

// order-preserving float <-> uint32 keys for atomic min/max
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unkey(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ uint32_t bin_init(int w) {
  const int f = w % kBinFields;
  return f == 0 ? 0u : (f < 4 ? fkey(1e34f) : fkey(-1e34f));
}

__device__ __forceinline__ float gmin(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float gmax(float a, float b) { return a < b ? b : a; }
// AABB::Area (src/BVH/AABB.h:122-129)
__device__ __forceinline__ float area3(const float mn[3], const float mx[3]) {
  const float e0 = __fsub_rn(mx[0], mn[0]), e1 = __fsub_rn(mx[1], mn[1]), e2 = __fsub_rn(mx[2], mn[2]);
  const float s = __fadd_rn(__fadd_rn(__fmul_rn(e0, e1), __fmul_rn(e0, e2)), __fmul_rn(e1, e2));
  return fmaxf(0.0f, s);
}
__device__ __forceinline__ float plane_at(float mn, float mx, int i) {
  const float len = __fsub_rn(mx, mn);
  const float off = __fdiv_rn((float)i, (float)kIntervals);
  return __fadd_rn(mn, __fmul_rn(len, off));
}
__device__ __forceinline__ float centroid(float lo, float hi) { return __fmul_rn(__fadd_rn(lo, hi), 0.5f); }
__device__ __forceinline__ float comp(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// Adds the warp's primitives (one per lane, those with `in`) to bins bin[0..2] of
// the three axes (-1: the axis has none). Consecutive primitives mostly lie close
// together, so an axis often has few bins in a warp, and one atomic per lane and
// field would serialise on them: a bin that holds kBinGroup lanes or more takes
// their seven values reduced over the warp, in one atomic each; the lanes left
// over add their own.
constexpr int kBinGroup = 6;
__device__ __forceinline__ void bin_warp(uint32_t* bins, const int bin[3], const float4& l, const float4& h, bool in) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t key[6] = {fkey(l.x), fkey(l.y), fkey(l.z), fkey(h.x), fkey(h.y), fkey(h.z)};
  unsigned have = 0;  // the lanes whose union `mine` holds
  uint32_t mine = 0;  // lane f < 7: field f of that union
#pragma unroll
  for (int a = 0; a < 3; a++) {
    unsigned rem = __ballot_sync(FULL, in && bin[a] >= 0);
    while (rem) {
      const int b0 = __shfl_sync(FULL, bin[a], __ffs(rem) - 1);
      const unsigned same = __ballot_sync(FULL, in && bin[a] == b0);
      if (__popc(same) < kBinGroup) break;
      if (same != have) {
        have = same;
        mine = (uint32_t)__popc(same);
        const bool member = (same >> lane) & 1u;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const uint32_t mn = __reduce_min_sync(FULL, member ? key[k] : 0xffffffffu);
          const uint32_t mx = __reduce_max_sync(FULL, member ? key[3 + k] : 0u);
          if (lane == 1 + k) mine = mn;
          if (lane == 4 + k) mine = mx;
        }
      }
      uint32_t* e = bins + (a * kIntervals + b0) * kBinFields + lane;
      if (lane == 0) atomicAdd(e, mine);
      else if (lane < 4) atomicMin(e, mine);
      else if (lane < 7) atomicMax(e, mine);
      rem &= ~same;
    }
    if ((rem >> lane) & 1u) {
      uint32_t* e = bins + (a * kIntervals + bin[a]) * kBinFields;
      atomicAdd(e, 1u);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        atomicMin(e + 1 + k, key[k]);
        atomicMax(e + 4 + k, key[3 + k]);
      }
    }
  }
}

// The interval of one primitive per axis.
__device__ __forceinline__ void intervals_of(const float* planes, const float4& l, const float4& h, int iv[3]) {
  const float c[3] = {centroid(l.x, h.x), centroid(l.y, h.y), centroid(l.z, h.z)};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    iv[a] = 0;
#pragma unroll
    for (int j = 0; j < kPlanes; j++) iv[a] += !(c[a] <= planes[a * kPlanes + j]);
  }
}

struct Cand {
  float cost;
  uint32_t lc, rc;
  float lmn[3], lmx[3], rmn[3], rmx[3];
};

// Lane l < 30 evaluates axis l / 10, plane l % 10 + 1; returns the winning
// lane (first lowest cost below 1e34) or 32 when no candidate qualifies. The
// left and right unions of an axis' ten planes are two scans over its ten lanes
// (a lane that walks all intervals reads 77 words and decodes 66 keys); they keep
// the walk's order, earlier intervals on the left, so that equal bounds give the
// same bits.
__device__ __forceinline__ int choose_split(const uint32_t* bins, int lane, Cand& c) {
  const unsigned FULL = 0xffffffffu;
  const int a = lane / kPlanes, k = lane % kPlanes;
  const bool in = lane < 3 * kPlanes;
  bool valid = false;
  c.cost = 0.0f;
  c.lc = c.rc = 0;
  for (int x = 0; x < 3; x++) c.lmn[x] = c.rmn[x] = 1e34f, c.lmx[x] = c.rmx[x] = -1e34f;
  if (in) {
    const uint32_t* e = bins + (a * kIntervals + k) * kBinFields;
    c.lc = e[0], c.rc = e[kBinFields];
    for (int x = 0; x < 3; x++) {
      c.lmn[x] = gmin(c.lmn[x], unkey(e[1 + x])), c.lmx[x] = gmax(c.lmx[x], unkey(e[4 + x]));
      c.rmn[x] = gmin(c.rmn[x], unkey(e[kBinFields + 1 + x])), c.rmx[x] = gmax(c.rmx[x], unkey(e[kBinFields + 4 + x]));
    }
  }
#pragma unroll
  for (int off = 1; off < kPlanes; off <<= 1) {
    const uint32_t ul = __shfl_up_sync(FULL, c.lc, off), dr = __shfl_down_sync(FULL, c.rc, off);
    const bool up = k >= off, down = k + off < kPlanes;
    if (up) c.lc += ul;
    if (down) c.rc += dr;
#pragma unroll
    for (int x = 0; x < 3; x++) {
      const float umn = __shfl_up_sync(FULL, c.lmn[x], off), umx = __shfl_up_sync(FULL, c.lmx[x], off);
      const float dmn = __shfl_down_sync(FULL, c.rmn[x], off), dmx = __shfl_down_sync(FULL, c.rmx[x], off);
      if (up) c.lmn[x] = gmin(umn, c.lmn[x]), c.lmx[x] = gmax(umx, c.lmx[x]);
      if (down) c.rmn[x] = gmin(c.rmn[x], dmn), c.rmx[x] = gmax(c.rmx[x], dmx);
    }
  }
  if (in) {
    c.cost = __fadd_rn(__fmul_rn(area3(c.lmn, c.lmx), __uint2float_rn(c.lc)),
                       __fmul_rn(area3(c.rmn, c.rmx), __uint2float_rn(c.rc)));
    valid = c.cost < 1e34f;
  }
  float bc = valid ? c.cost : 0.0f;
  int bl = valid ? lane : 32;
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, bc, off);
    const int ol = __shfl_xor_sync(0xffffffffu, bl, off);
    if (ol < 32 && (bl == 32 || oc < bc || (oc == bc && ol < bl))) bc = oc, bl = ol;
  }
  return bl;
}

__device__ __forceinline__ void bcast_cand(Cand& c, int src) {
  c.cost = __shfl_sync(0xffffffffu, c.cost, src);
  c.lc = __shfl_sync(0xffffffffu, c.lc, src);
  c.rc = __shfl_sync(0xffffffffu, c.rc, src);
  for (int k = 0; k < 3; k++) {
    c.lmn[k] = __shfl_sync(0xffffffffu, c.lmn[k], src);
    c.lmx[k] = __shfl_sync(0xffffffffu, c.lmx[k], src);
    c.rmn[k] = __shfl_sync(0xffffffffu, c.rmn[k], src);
    c.rmx[k] = __shfl_sync(0xffffffffu, c.rmx[k], src);
  }
}

__device__ __forceinline__ BNode make_node(const float mn[3], const float mx[3], uint32_t first, uint32_t count,
                                           int32_t parent, int32_t depth) {
  BNode b;
  for (int k = 0; k < 3; k++) b.mn[k] = mn[k], b.mx[k] = mx[k];
  b.first = (int32_t)first;
  b.count = (int32_t)count;
  b.left = -1;
  b.parent = parent;
  b.depth = depth;
  b.qcount = 0;
  return b;
}

// ---------------------------------------------------------------- prep
__global__ void k_init(uint32_t* counters) {
  const int w = threadIdx.x;
  if (w < kCounterWords)
    counters[w] = (w >= kRootKeys && w < kRootKeys + 3) ? fkey(1e34f)
                  : (w >= kRootKeys + 3 && w < kRootKeys + 6) ? fkey(-1e34f)
                                                              : 0u;
}

// Root bounds: reduced over the block before the six counters every block shares
// are touched. With one atomic per warp the 2.0 M-triangle prep spent 290 of its
// us on them.
__device__ __forceinline__ void block_root_keys(uint32_t* counters, uint32_t kmn[3], uint32_t kmx[3]) {
  __shared__ uint32_t red[6];
  if (threadIdx.x < 6) red[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  for (int k = 0; k < 3; k++) {
    kmn[k] = __reduce_min_sync(0xffffffffu, kmn[k]);
    kmx[k] = __reduce_max_sync(0xffffffffu, kmx[k]);
  }
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 3; k++) atomicMin(&red[k], kmn[k]), atomicMax(&red[3 + k], kmx[k]);
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(&counters[kRootKeys + threadIdx.x], red[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&counters[kRootKeys + threadIdx.x], red[threadIdx.x]);
}

// prims: the buffer of the first level, or the final one when the root is small
__global__ void __launch_bounds__(256) k_prep(const float4* __restrict__ v, const uint4* __restrict__ idx, uint32_t n,
                                              PrimBox* __restrict__ box,
                                              uint32_t* __restrict__ prims, uint32_t* counters) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t kmn[3] = {fkey(1e34f), fkey(1e34f), fkey(1e34f)}, kmx[3] = {fkey(-1e34f), fkey(-1e34f), fkey(-1e34f)};
  if (i < n) {
    const uint4 t = idx[i];
    const float4 a = v[t.x], b = v[t.y], c = v[t.z];
    // triangle::getBounds (src/Core/Triangle.cuh:59-65): min - 0.001, max + 0.01
    const float plo = 0.001f, phi = 0.01f;
    const float mn[3] = {__fsub_rn(gmin(a.x, gmin(b.x, c.x)), plo), __fsub_rn(gmin(a.y, gmin(b.y, c.y)), plo),
                         __fsub_rn(gmin(a.z, gmin(b.z, c.z)), plo)};
    const float mx[3] = {__fadd_rn(gmax(a.x, gmax(b.x, c.x)), phi), __fadd_rn(gmax(a.y, gmax(b.y, c.y)), phi),
                         __fadd_rn(gmax(a.z, gmax(b.z, c.z)), phi)};
    box[i] = PrimBox{make_float4(mn[0], mn[1], mn[2], 0.0f), make_float4(mx[0], mx[1], mx[2], 0.0f)};
    prims[i] = i;
    for (int k = 0; k < 3; k++) kmn[k] = fkey(mn[k]), kmx[k] = fkey(mx[k]);
  }
  block_root_keys(counters, kmn, kmx);
}

__global__ void k_root(BNode* arena, int32_t* large, int32_t* mid, int32_t* small, uint32_t n, uint32_t mid_most,
                       uint32_t* counters) {
  float mn[3], mx[3];
  for (int k = 0; k < 3; k++) mn[k] = unkey(counters[kRootKeys + k]), mx[k] = unkey(counters[kRootKeys + 3 + k]);
  arena[0] = make_node(mn, mx, 0, n, -1, 0);
  counters[kArenaCount] = 1;
  if (n >= 4) {
    if (n > mid_most) {
      large[0] = 0;
      counters[kLarge] = 1;
    } else if (n > kWarpMax) {
      mid[0] = 0;
      counters[kMid] = 1;
    } else {
      small[0] = 0;
      counters[kSmallCount] = 1;
    }
  }
}

// ---------------------------------------------------------------- large nodes, one level
// The kernels of a level read how many nodes and chunks it has from the counters of
// its parity, so that several levels can be issued without asking the device (their
// grids are upper bounds). A large node's primitives lie in the buffer of its
// level's parity; the partition writes those of its children to the other one when
// they are large and to the final array otherwise, so nothing is copied back.
struct LevelArgs {
  BNode* arena;
  int32_t* large[2];
  uint32_t max_large;
  int32_t* mid;
  uint32_t max_mid, mid_most;
  int32_t* small;
  uint32_t* counters;
  uint32_t cap;
  uint32_t chunk, max_chunks;
  Chunk* chunks;
  Split* split;
  uint32_t* bins;
  uint32_t* chunk_left;
  uint32_t* left;  // a bit per primitive of a chunk: goes left (chunk / 32 words each)
  const PrimBox* box;
  uint32_t* buf[2];
  uint32_t* prims;
};
__device__ __forceinline__ uint32_t large_count(const LevelArgs& A, int par) {
  return min(A.counters[kLarge + par], A.max_large);
}
__device__ __forceinline__ uint32_t chunk_count(const LevelArgs& A, int par) {
  return min(A.counters[kChunks + par], A.max_chunks);
}

// One warp per node: its lanes write the chunks and the empty bins.
__global__ void __launch_bounds__(256) k_chunks(LevelArgs A, int par) {
  after_previous();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  // the next level's counters: its last reader was the level before this one
  if (blockIdx.x == 0 && threadIdx.x == 0) A.counters[kLarge + (par ^ 1)] = 0, A.counters[kChunks + (par ^ 1)] = 0;
  if (s >= large_count(A, par)) return;  // whole warp
  const BNode& nd = A.arena[A.large[par][s]];
  const uint32_t cnt = (uint32_t)nd.count, nc = (cnt + A.chunk - 1) / A.chunk;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&A.counters[kChunks + par], nc);
  base = __shfl_sync(0xffffffffu, base, 0);
  for (uint32_t c = lane; c < nc; c += 32) {
    const uint32_t b = (uint32_t)nd.first + c * A.chunk;
    if (base + c < A.max_chunks)  // always: the ranges are disjoint
      A.chunks[base + c] = Chunk{(int32_t)s, b, (uint32_t)nd.first + min(cnt, (c + 1) * A.chunk)};
  }
  if (lane == 0) A.split[s] = Split{-1, 0.0f, 0u, base, 0u};
  uint32_t* b = A.bins + (size_t)s * kBinWords;
  for (int w = lane; w < kBinWords; w += 32) b[w] = bin_init(w);
}

__global__ void __launch_bounds__(256) k_bin(LevelArgs A, int par) {
  after_previous();
  __shared__ float planes[3 * kPlanes];
  __shared__ uint32_t bins[kBinWords];
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const BNode& nd = A.arena[A.large[par][ch.slot]];
  const uint32_t* prims = A.buf[par];
  if (threadIdx.x < 3 * kPlanes) {
    const int a = threadIdx.x / kPlanes, i = threadIdx.x % kPlanes + 1;
    planes[threadIdx.x] = plane_at(nd.mn[a], nd.mx[a], i);
  }
  for (int w = threadIdx.x; w < kBinWords; w += blockDim.x) bins[w] = bin_init(w);
  __syncthreads();
  for (uint32_t k0 = ch.begin; k0 < ch.end; k0 += blockDim.x) {
    const bool in = k0 + threadIdx.x < ch.end;
    const PrimBox v = prim_box(A.box + (in ? prims[k0 + threadIdx.x] : 0u));
    int iv[3];
    intervals_of(planes, v.lo, v.hi, iv);
    bin_warp(bins, iv, v.lo, v.hi, in);
  }
  __syncthreads();
  uint32_t* g = A.bins + (size_t)ch.slot * kBinWords;
  for (int w = threadIdx.x; w < kBinWords; w += blockDim.x) {
    const uint32_t v = bins[w];
    const int f = w % kBinFields;
    if (f == 0) {
      if (v) atomicAdd(&g[w], v);
    } else if (f < 4) {
      if (v != fkey(1e34f)) atomicMin(&g[w], v);
    } else {
      if (v != fkey(-1e34f)) atomicMax(&g[w], v);
    }
  }
}

// Queue of a child that a block or a warp splits further.
__device__ __forceinline__ void queue_child(const LevelArgs& A, int32_t id, uint32_t count, int32_t depth) {
  if (count < 4 || depth > kMaxSplitDepth) return;  // a leaf
  if (count > kWarpMax) {
    const uint32_t s = atomicAdd(&A.counters[kMid], 1u);
    if (s < A.max_mid) A.mid[s] = id;  // always: the ranges are disjoint
    return;
  }
  A.small[atomicAdd(&A.counters[kSmallCount], 1u)] = id;
}

// Place a new child: on the next level (true), or with queue_child.
__device__ __forceinline__ bool classify(const LevelArgs& A, int par, int32_t id, uint32_t count, int32_t depth) {
  if (count <= A.mid_most || depth > kMaxSplitDepth) {
    queue_child(A, id, count, depth);
    return false;
  }
  const uint32_t s = atomicAdd(&A.counters[kLarge + (par ^ 1)], 1u);
  if (s < A.max_large) A.large[par ^ 1][s] = id;
  return s < A.max_large;
}

__global__ void __launch_bounds__(256) k_split(LevelArgs A, int par) {
  after_previous();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (s >= large_count(A, par)) return;  // whole warp
  const int32_t ni = A.large[par][s];
  const BNode nd = A.arena[ni];
  // the candidates walk the bins word by word: from shared memory
  __shared__ uint32_t sbins[8][kBinWords];
  uint32_t* bins = sbins[threadIdx.x >> 5];
  for (int w = lane; w < kBinWords; w += 32) bins[w] = A.bins[(size_t)s * kBinWords + w];
  __syncwarp();
  Cand c;
  const int best = choose_split(bins, lane, c);
  const float parent_cost = __fmul_rn(area3(nd.mn, nd.mx), __uint2float_rn((uint32_t)nd.count));
  if (best == 32) {
    // no candidate below 1e34: a leaf unless the parent's cost is not below it either
    if (!(parent_cost < 1e34f) && lane == 0) atomicOr(&A.counters[kError], kErrDegenerate);
    return;
  }
  bcast_cand(c, best);
  if (parent_cost < c.cost) return;
  if (lane != 0) return;
  const int a = best / kPlanes, i = best % kPlanes + 1;
  const uint32_t cid = atomicAdd(&A.counters[kArenaCount], 2u);
  if (cid + 2 > A.cap) {
    atomicOr(&A.counters[kError], kErrArena);
    return;
  }
  A.arena[cid] = make_node(c.lmn, c.lmx, (uint32_t)nd.first, c.lc, ni, nd.depth + 1);
  A.arena[cid + 1] = make_node(c.rmn, c.rmx, (uint32_t)nd.first + c.lc, c.rc, ni, nd.depth + 1);
  A.arena[ni].left = (int32_t)cid;
  uint32_t queued = classify(A, par, (int32_t)cid, c.lc, nd.depth + 1) ? 1u : 0u;
  queued |= classify(A, par, (int32_t)cid + 1, c.rc, nd.depth + 1) ? 2u : 0u;
  A.split[s] = Split{a, plane_at(nd.mn[a], nd.mx[a], i), c.lc, A.split[s].chunk0, queued};
}

__device__ __forceinline__ bool goes_left(const PrimBox* box, uint32_t p, int axis, float coord) {
  const PrimBox v = prim_box(box + p);
  return centroid(comp(v.lo, axis), comp(v.hi, axis)) <= coord;
}

// Which side each primitive of a chunk goes to (a bit each), and how many go left.
__global__ void __launch_bounds__(256) k_part_count(LevelArgs A, int par) {
  after_previous();
  __shared__ uint32_t nleft;
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const Split sp = A.split[ch.slot];
  if (sp.axis < 0) return;
  const uint32_t* prims = A.buf[par];
  if (threadIdx.x == 0) nleft = 0;
  __syncthreads();
  uint32_t n = 0;
  uint32_t* bits = A.left + (size_t)blockIdx.x * (A.chunk / 32);
  for (uint32_t k0 = ch.begin; k0 < ch.end; k0 += blockDim.x) {
    const uint32_t k = k0 + threadIdx.x;
    const uint32_t b = __ballot_sync(0xffffffffu, k < ch.end && goes_left(A.box, prims[k], sp.axis, sp.coord));
    if ((threadIdx.x & 31) == 0) bits[(k0 - ch.begin + threadIdx.x) / 32] = b, n += __popc(b);
  }
  if (n) atomicAdd(&nleft, n);
  __syncthreads();
  if (threadIdx.x == 0) A.chunk_left[blockIdx.x] = nleft;
}

// Stable partition by k_part_count's bits; every block adds up the node's chunk
// counts before its own. A node that stays a leaf goes to the final array as it
// lies, and so does a range whose counts don't give the split's left count (they
// come from the same bins; the build fails).
constexpr int kMaxWords = 2048 / 32;  // bit words of a chunk
__global__ void __launch_bounds__(256) k_part_scatter(LevelArgs A, int par) {
  after_previous();
  __shared__ uint32_t word[kMaxWords], before[kMaxWords], sum[2];
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const Split sp = A.split[ch.slot];
  const uint32_t* from = A.buf[par];
  if (sp.axis < 0) {
    for (uint32_t k = ch.begin + threadIdx.x; k < ch.end; k += blockDim.x) A.prims[k] = from[k];
    return;
  }
  const BNode& nd = A.arena[A.large[par][ch.slot]];
  const uint32_t first = (uint32_t)nd.first, nc = ((uint32_t)nd.count + A.chunk - 1) / A.chunk;
  const uint32_t mine = blockIdx.x - sp.chunk0, cnt = ch.end - ch.begin, words = (cnt + 31) / 32;
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  uint32_t pre = 0, all = 0;
  for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x) {
    const uint32_t v = A.chunk_left[sp.chunk0 + c];
    all += v;
    if (c < mine) pre += v;
  }
  pre = __reduce_add_sync(0xffffffffu, pre), all = __reduce_add_sync(0xffffffffu, all);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0 && all) atomicAdd(&sum[0], pre), atomicAdd(&sum[1], all);
  if (warp == 0) {  // left counts before each word
    uint32_t run = 0;
    for (uint32_t w0 = 0; w0 < words; w0 += 32) {
      const uint32_t w = w0 + lane, b = w < words ? A.left[(size_t)blockIdx.x * (A.chunk / 32) + w] : 0u;
      const uint32_t v = __popc(b);
      uint32_t x = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
      }
      if (w < words) word[w] = b, before[w] = run + x - v;
      run += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  __syncthreads();
  uint32_t* to_l = sp.queued & 1u ? A.buf[par ^ 1] : A.prims;
  uint32_t* to_r = sp.queued & 2u ? A.buf[par ^ 1] : A.prims;
  if (sum[1] != sp.lc) {
    if (threadIdx.x == 0) atomicOr(&A.counters[kError], kErrPartition);
    for (uint32_t k = ch.begin + threadIdx.x; k < ch.end; k += blockDim.x)
      (k < first + sp.lc ? to_l : to_r)[k] = from[k];
    return;
  }
  const uint32_t dl = first + sum[0], dr = first + sp.lc + (ch.begin - first) - sum[0];
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t w = warp; w < words; w += 8) {
    if (32 * w + lane >= cnt) continue;
    const uint32_t b = word[w], l = before[w] + __popc(b & lt), p = from[ch.begin + 32 * w + lane];
    if ((b >> lane) & 1u) to_l[dl + l] = p;
    else to_r[dr + 32 * w + lane - l] = p;
  }
}

// ---------------------------------------------------------------- nodes of at most mid_size(n), one block each
// A block splits such a node, and its children of more than kWarpMax primitives, with
// everything in shared memory: boxes and ids by the slot they arrived in, and the
// slots in their present order, in two arrays that a partition goes between. A node
// that stays a leaf, and children of at most kWarpMax, go to the final array. The
// level kernels would take five launches a level for them: 20,480 triangles 528 -> 496
// us, 2.0 M 3.09 -> 2.92 ms.
struct MidNode {
  int32_t node, depth;
  uint32_t first, count;  // first: within the block's range
  uint32_t par;           // which array its slots lie in
  float mn[3], mx[3];
};
struct MidSplit {
  int32_t axis;  // -1: the node stays a leaf
  float coord;
  uint32_t lc;
  int32_t kid[2];  // the children's places on the stack, -1 where they have none
};
constexpr size_t kMidBytes = (6 * sizeof(float) + sizeof(uint32_t) + 2 * sizeof(uint16_t));  // per primitive

template <uint32_t kMidMax, int kMidThreads>
__global__ void __launch_bounds__(kMidThreads) k_mid(LevelArgs A) {
  after_previous();
  constexpr uint32_t kMidWords = kMidMax / 32;
  constexpr int kMidStack = kMidMax / (kWarpMax + 1) + 1;  // pending nodes are disjoint
  extern __shared__ float sh[];
  float* bx = sh;  // bx[c * kMidMax + slot]: min x/y/z, max x/y/z
  uint32_t* id = reinterpret_cast<uint32_t*>(bx + 6 * kMidMax);
  uint16_t* ord = reinterpret_cast<uint16_t*>(id + kMidMax);  // two arrays
  __shared__ uint32_t bins[kBinWords];
  __shared__ float planes[3 * kPlanes];
  __shared__ MidNode stack[kMidStack];
  __shared__ MidSplit split;
  __shared__ uint32_t wleft[kMidWords], before[kMidWords], total;
  __shared__ int s_sp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t nmid = min(A.counters[kMid], A.max_mid);
  for (uint32_t m = blockIdx.x; m < nmid; m += gridDim.x) {
    const int32_t root = A.mid[m];
    const uint32_t base = (uint32_t)A.arena[root].first, n = (uint32_t)A.arena[root].count;
    if (threadIdx.x == 0) {
      stack[0].node = root, stack[0].depth = A.arena[root].depth;
      stack[0].first = 0, stack[0].count = n, stack[0].par = 0;
      for (int a = 0; a < 3; a++) stack[0].mn[a] = A.arena[root].mn[a], stack[0].mx[a] = A.arena[root].mx[a];
    }
    for (int w = threadIdx.x; w < kBinWords; w += kMidThreads) bins[w] = bin_init(w);
    for (uint32_t j = threadIdx.x; j < n; j += kMidThreads) {
      const uint32_t p = A.prims[base + j];
      const PrimBox v = prim_box(A.box + p);
      id[j] = p, ord[j] = (uint16_t)j;
      bx[j] = v.lo.x, bx[kMidMax + j] = v.lo.y, bx[2 * kMidMax + j] = v.lo.z;
      bx[3 * kMidMax + j] = v.hi.x, bx[4 * kMidMax + j] = v.hi.y, bx[5 * kMidMax + j] = v.hi.z;
    }
    __syncthreads();
    int sp = 1;
    while (sp > 0) {
      const MidNode nd = stack[--sp];
      const uint32_t first = nd.first, count = nd.count;
      const uint16_t* from = ord + nd.par * kMidMax;
      if (threadIdx.x < 3 * kPlanes) {
        const int a = threadIdx.x / kPlanes, i = threadIdx.x % kPlanes + 1;
        planes[threadIdx.x] = plane_at(nd.mn[a], nd.mx[a], i);
      }
      __syncthreads();
      for (uint32_t k0 = 0; k0 + 32 * warp < count; k0 += kMidThreads) {
        const uint32_t k = k0 + threadIdx.x;
        const bool in = k < count;
        const uint32_t j = in ? from[first + k] : 0u;
        const float4 lo = make_float4(bx[j], bx[kMidMax + j], bx[2 * kMidMax + j], 0.0f);
        const float4 hi = make_float4(bx[3 * kMidMax + j], bx[4 * kMidMax + j], bx[5 * kMidMax + j], 0.0f);
        int iv[3];
        intervals_of(planes, lo, hi, iv);
        bin_warp(bins, iv, lo, hi, in);
      }
      __syncthreads();
      if (warp == 0) {
        Cand c;
        const int best = choose_split(bins, lane, c);
        const float parent_cost = __fmul_rn(area3(nd.mn, nd.mx), __uint2float_rn(count));
        if (best < 32) bcast_cand(c, best);
        if (lane == 0) {
          split = MidSplit{-1, 0.0f, 0u, {-1, -1}};
          int top = sp;
          if (best == 32) {
            // no candidate below 1e34: a leaf unless the parent's cost is not below it either
            if (!(parent_cost < 1e34f)) atomicOr(&A.counters[kError], kErrDegenerate);
          } else if (!(parent_cost < c.cost)) {
            const uint32_t cid = atomicAdd(&A.counters[kArenaCount], 2u);
            if (cid + 2 > A.cap) {
              atomicOr(&A.counters[kError], kErrArena);
            } else {
              const uint32_t g = base + first;
              split.axis = best / kPlanes, split.coord = planes[best], split.lc = c.lc;
              A.arena[cid] = make_node(c.lmn, c.lmx, g, c.lc, nd.node, nd.depth + 1);
              A.arena[cid + 1] = make_node(c.rmn, c.rmx, g + c.lc, c.rc, nd.node, nd.depth + 1);
              A.arena[nd.node].left = (int32_t)cid;
              for (int i = 0; i < 2; i++) {
                const uint32_t cc = i ? c.rc : c.lc;
                if (cc > kWarpMax && nd.depth + 1 <= kMaxSplitDepth) {
                  split.kid[i] = top;  // at most kMidStack pending: ranges of more than kWarpMax, disjoint
                  MidNode& q = stack[top++];
                  q.node = (int32_t)cid + i, q.depth = nd.depth + 1;
                  q.first = first + (i ? c.lc : 0u), q.count = cc, q.par = nd.par ^ 1u;
                  for (int a = 0; a < 3; a++)
                    q.mn[a] = i ? c.rmn[a] : c.lmn[a], q.mx[a] = i ? c.rmx[a] : c.lmx[a];
                } else {
                  queue_child(A, (int32_t)cid + i, cc, nd.depth + 1);
                }
              }
            }
          }
          s_sp = top;
        }
      }
      __syncthreads();
      sp = s_sp;
      for (int w = threadIdx.x; w < kBinWords; w += kMidThreads) bins[w] = bin_init(w);
      const MidSplit s = split;
      if (s.axis < 0) {
        for (uint32_t k = threadIdx.x; k < count; k += kMidThreads) A.prims[base + first + k] = id[from[first + k]];
        __syncthreads();
        continue;
      }
      // the stable partition: a bit per primitive, kept in the lane that read it
      uint32_t slot[kMidMax / kMidThreads], bal[kMidMax / kMidThreads];
#pragma unroll
      for (int i = 0; i < (int)(kMidMax / kMidThreads); i++) {
        const uint32_t w = warp + (kMidThreads / 32) * i, k = 32 * w + lane;
        if (32 * w >= count) break;  // whole warp
        slot[i] = k < count ? from[first + k] : 0u;
        const float c = centroid(bx[s.axis * kMidMax + slot[i]], bx[(3 + s.axis) * kMidMax + slot[i]]);
        bal[i] = __ballot_sync(0xffffffffu, k < count && c <= s.coord);
        if (lane == 0) wleft[w] = __popc(bal[i]);
      }
      __syncthreads();
      if (warp == 0) {  // left counts before each word
        uint32_t run = 0;
        for (uint32_t w0 = 0; 32 * w0 < count; w0 += 32) {
          const uint32_t w = w0 + lane, v = 32 * w < count ? wleft[w] : 0u;
          uint32_t x = v;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
          }
          if (32 * w < count) before[w] = run + x - v;
          run += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) total = run;
      }
      __syncthreads();
      const bool good = total == s.lc;
      if (!good && threadIdx.x == 0) atomicOr(&A.counters[kError], kErrPartition);
      uint16_t* to = ord + (nd.par ^ 1u) * kMidMax;
#pragma unroll
      for (int i = 0; i < (int)(kMidMax / kMidThreads); i++) {
        const uint32_t w = warp + (kMidThreads / 32) * i, k = 32 * w + lane;
        if (k >= count) break;
        const uint32_t l = before[w] + __popc(bal[i] & lt);
        bool left = (bal[i] >> lane) & 1u;
        uint32_t at = first + (left ? l : s.lc + k - l);
        if (!good) left = k < s.lc, at = first + k;  // as it lies; the build fails
        if ((left ? s.kid[0] : s.kid[1]) >= 0) to[at] = (uint16_t)slot[i];
        else A.prims[base + at] = id[slot[i]];
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- small subtrees, one warp each
// tasks: ranges of 4..kLeafTask primitives for k_leaf, counted in counters[kTasks]
// (disjoint, so at most n / 4).
__global__ void __launch_bounds__(kSmallWarps * 32) k_small(BNode* arena, const int32_t* __restrict__ small,
                                                            const uint32_t* counters_ro,
                                                            const PrimBox* __restrict__ box, uint32_t* prims,
                                                            uint32_t* counters, uint32_t cap, uint32_t* tasks) {
  __shared__ uint32_t sbins[kSmallWarps][kBinWords];
  __shared__ float splanes[kSmallWarps][3 * kPlanes];
  __shared__ int32_t sstack[kSmallWarps][kSmallStack];
  __shared__ uint32_t stmp[kSmallWarps][2 * kWarpMax];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* bins = sbins[warp];
  float* planes = splanes[warp];
  int32_t* stack = sstack[warp];
  uint32_t* tmp = stmp[warp];
  const uint32_t nsmall = counters_ro[kSmallCount];
  for (uint32_t s = blockIdx.x * kSmallWarps + warp; s < nsmall; s += gridDim.x * kSmallWarps) {
    const int32_t root = small[s];
    if ((uint32_t)arena[root].count <= kLeafTask) {
      if (lane == 0) tasks[atomicAdd(&counters[kTasks], 1u)] = (uint32_t)root;
      continue;
    }
    if (lane == 0) stack[0] = root;
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
      const int32_t ni = stack[--sp];
      __syncwarp();
      const BNode nd = arena[ni];
      const uint32_t first = (uint32_t)nd.first, count = (uint32_t)nd.count;
      if (lane < 3 * kPlanes) planes[lane] = plane_at(nd.mn[lane / kPlanes], nd.mx[lane / kPlanes], lane % kPlanes + 1);
      for (int w = lane; w < kBinWords; w += 32) bins[w] = bin_init(w);
      __syncwarp();
      for (uint32_t k0 = 0; k0 < count; k0 += 32) {
        const bool in = k0 + lane < count;
        const PrimBox v = prim_box(box + (in ? prims[first + k0 + lane] : 0u));
        int iv[3];
        intervals_of(planes, v.lo, v.hi, iv);
        bin_warp(bins, iv, v.lo, v.hi, in);
      }
      __syncwarp();
      Cand c;
      const int best = choose_split(bins, lane, c);
      const float parent_cost = __fmul_rn(area3(nd.mn, nd.mx), __uint2float_rn(count));
      if (best == 32) {
        if (!(parent_cost < 1e34f) && lane == 0) atomicOr(&counters[kError], kErrDegenerate);
        continue;
      }
      bcast_cand(c, best);
      if (parent_cost < c.cost) continue;
      const int a = best / kPlanes;
      const float coord = planes[best];
      // stable partition through shared memory
      uint32_t nl = 0, nr = 0;
      for (uint32_t k0 = 0; k0 < count; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool in = k < count;
        const uint32_t p = in ? prims[first + k] : 0u;
        const bool left = in && goes_left(box, p, a, coord);
        const uint32_t bl = __ballot_sync(0xffffffffu, left), br = __ballot_sync(0xffffffffu, in && !left);
        if (left) tmp[nl + __popc(bl & lt)] = p;
        else if (in) tmp[kWarpMax + nr + __popc(br & lt)] = p;
        nl += __popc(bl), nr += __popc(br);
      }
      __syncwarp();
      if (nl != c.lc) {
        if (lane == 0) atomicOr(&counters[kError], kErrPartition);
        continue;
      }
      for (uint32_t k = lane; k < count; k += 32) prims[first + k] = k < nl ? tmp[k] : tmp[kWarpMax + k - nl];
      uint32_t cid = 0;
      if (lane == 0) cid = atomicAdd(&counters[kArenaCount], 2u);
      cid = __shfl_sync(0xffffffffu, cid, 0);
      if (cid + 2 > cap) {
        if (lane == 0) atomicOr(&counters[kError], kErrArena);
        continue;
      }
      if (lane == 0) {
        arena[cid] = make_node(c.lmn, c.lmx, first, c.lc, ni, nd.depth + 1);
        arena[cid + 1] = make_node(c.rmn, c.rmx, first + c.lc, c.rc, ni, nd.depth + 1);
        arena[ni].left = (int32_t)cid;
      }
      const bool more_r = c.rc >= 4 && nd.depth + 1 <= kMaxSplitDepth;
      const bool more_l = c.lc >= 4 && nd.depth + 1 <= kMaxSplitDepth;
      const bool task_r = more_r && c.rc <= kLeafTask, task_l = more_l && c.lc <= kLeafTask;
      const bool push_r = more_r && !task_r, push_l = more_l && !task_l;
      if (lane == 0 && (task_l || task_r)) {
        uint32_t at_ = atomicAdd(&counters[kTasks], (uint32_t)task_l + (uint32_t)task_r);
        if (task_l) tasks[at_++] = cid;
        if (task_r) tasks[at_] = cid + 1;
      }
      if (sp + (int)push_r + (int)push_l > kSmallStack) {
        if (lane == 0) atomicOr(&counters[kError], kErrStack);
        continue;
      }
      if (lane == 0) {
        if (push_r) stack[sp] = (int32_t)cid + 1;
        if (push_l) stack[sp + (int)push_r] = (int32_t)cid;
      }
      sp += (int)push_r + (int)push_l;
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- subtrees of at most kLeafTask primitives, one thread each
// The SAH of k_small by one thread for a whole subtree, 32 of them per warp. The
// range is sorted once per axis by centroid; an order is 16 nibbles of a 64-bit
// word, and a split partitions every order stably. A plane's left primitives
// are then a prefix of its axis' order, so the ten planes of an axis cost one
// suffix pass (areas) and one prefix walk. `cur` is the range's own order, which
// the stable partition of k_small would leave. Boxes lie in shared memory
// [value][thread], free of bank conflicts whatever primitive a thread reads.
// Splits are found first, so the arena is asked for the nodes that exist.
//
// One warp per node spent its shuffles and 231 bin words on four primitives as
// on 128: k_small took 2.69 ms of a 2.0 M-triangle build; with the leaves here it
// takes 0.55 and this kernel 0.57 ms.
// Few tasks are spread over all resident warps, a few lanes each: a warp is as slow
// as its lanes' different paths added up (20,480 triangles: 158 us with 32 tasks to
// a warp, 96 spread).
constexpr int kLeafThreads = 64;
// boxes, centroids or right areas, ids, nodes: a node of 4 or more splits, so 16
// primitives make at most 13 splits and 27 nodes
constexpr int kLeafWords = 16 * 6 + 16 + 16 + 27;
constexpr size_t kLeafShared = sizeof(float) * kLeafWords * kLeafThreads;

__device__ __forceinline__ uint32_t nib(unsigned long long o, uint32_t i) { return (uint32_t)(o >> (4 * i)) & 15u; }
// Positions b..b+n-1 of order o, those of `left` first, each part in its order.
__device__ __forceinline__ unsigned long long part_order(unsigned long long o, uint32_t b, uint32_t n, uint32_t nl,
                                                         uint32_t left) {
  const unsigned long long src = o;
  uint32_t pl = b, pr = b + nl;
  for (uint32_t i = 0; i < n; i++) {
    const uint32_t j = nib(src, b + i);
    const uint32_t to = (left >> j) & 1u ? pl++ : pr++;
    o = (o & ~(15ull << (4 * to))) | ((unsigned long long)j << (4 * to));
  }
  return o;
}

__global__ void __launch_bounds__(kLeafThreads) k_leaf(BNode* arena, const uint32_t* __restrict__ tasks,
                                                       const PrimBox* __restrict__ boxes,
                                                       uint32_t* prims, uint32_t* counters, uint32_t cap) {
  extern __shared__ float sh[];
  constexpr int T = kLeafThreads;
  float* box = sh + threadIdx.x;                           // box[(6 j + c) T]: min x/y/z, max x/y/z of primitive j
  float* val = box + 96 * T;                               // val[i T]: centroids while sorting, then right areas
  uint32_t* id = reinterpret_cast<uint32_t*>(val + 16 * T);  // id[j T]
  uint32_t* node = id + 16 * T;  // node k (k-th made): b | n << 4 | left count << 9 | depth << 14
  const uint32_t ntask = counters[kTasks];
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (T / 32), lanes = min(32u, (ntask + warps - 1) / warps);
  for (uint32_t t0 = (blockIdx.x * (T / 32) + (threadIdx.x >> 5)) * lanes; t0 < ntask; t0 += warps * lanes) {
    const bool in = lane < (int)lanes && t0 + lane < ntask;
    const int32_t root = in ? (int32_t)tasks[t0 + lane] : 0;
    uint32_t first = 0, count = 0, splits = 0;
    int32_t depth0 = 0;
    unsigned long long ord[3] = {0, 0, 0}, cur = 0xfedcba9876543210ull;
    if (in) {
      const BNode nd = arena[root];
      first = (uint32_t)nd.first, count = (uint32_t)nd.count, depth0 = nd.depth;
      for (uint32_t j = 0; j < count; j++) {
        const uint32_t p = prims[first + j];
        const PrimBox v = prim_box(boxes + p);
        const float4 l = v.lo, h = v.hi;
        float* b = box + 6 * j * T;
        b[0] = l.x, b[T] = l.y, b[2 * T] = l.z, b[3 * T] = h.x, b[4 * T] = h.y, b[5 * T] = h.z;
        id[j * T] = p;
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        unsigned long long o = 0;
        for (uint32_t j = 0; j < count; j++) {  // insertion: o's nibbles 0..j-1 are sorted
          const float c = centroid(box[(6 * j + a) * T], box[(6 * j + 3 + a) * T]);
          val[j * T] = c;
          uint32_t k = j;
          while (k > 0 && !(val[nib(o, k - 1) * T] <= c)) k--;
          const unsigned long long low = o & ((1ull << (4 * k)) - 1ull);
          o = low | ((unsigned long long)j << (4 * k)) | ((o - low) << 4);
        }
        ord[a] = o;
      }
      node[0] = count << 4;
      // nodes in the order they are made; the two children of the k-th split are nodes 2 k + 1 and 2 k + 2
      for (uint32_t k = 0; k <= 2 * splits; k++) {
        const uint32_t w = node[k * T], b = w & 15u, n = (w >> 4) & 31u, dep = w >> 14;
        if (n < 4 || depth0 + (int32_t)dep > kMaxSplitDepth) continue;
        float nmn[3] = {1e34f, 1e34f, 1e34f}, nmx[3] = {-1e34f, -1e34f, -1e34f};
        for (uint32_t i = 0; i < n; i++) {
          const float* q = box + 6 * nib(cur, b + i) * T;
          for (int c = 0; c < 3; c++) nmn[c] = fminf(nmn[c], q[c * T]), nmx[c] = fmaxf(nmx[c], q[(3 + c) * T]);
        }
        const float parent_cost = __fmul_rn(area3(nmn, nmx), __uint2float_rn(n));
        float best = 1e34f, coord = 0.0f;
        int bax = -1;
        uint32_t blc = 0;
        for (int a = 0; a < 3; a++) {
          const unsigned long long o = (a == 0 ? ord[0] : a == 1 ? ord[1] : ord[2]) >> (4 * b);
          float mn[3] = {1e34f, 1e34f, 1e34f}, mx[3] = {-1e34f, -1e34f, -1e34f};
          for (uint32_t i = n - 1; i > 0; i--) {
            const float* q = box + 6 * nib(o, i) * T;
            for (int c = 0; c < 3; c++) mn[c] = fminf(mn[c], q[c * T]), mx[c] = fmaxf(mx[c], q[(3 + c) * T]);
            val[i * T] = area3(mn, mx);
          }
          for (int c = 0; c < 3; c++) mn[c] = 1e34f, mx[c] = -1e34f;
          const float pmn = a == 0 ? nmn[0] : a == 1 ? nmn[1] : nmn[2], pmx = a == 0 ? nmx[0] : a == 1 ? nmx[1] : nmx[2];
          uint32_t lc = 0;
          for (int i = 1; i <= kPlanes; i++) {
            const float plane = plane_at(pmn, pmx, i);
            while (lc < n) {
              const float* q = box + 6 * nib(o, lc) * T;
              if (!(centroid(q[a * T], q[(3 + a) * T]) <= plane)) break;
              for (int c = 0; c < 3; c++) mn[c] = fminf(mn[c], q[c * T]), mx[c] = fmaxf(mx[c], q[(3 + c) * T]);
              lc++;
            }
            // an empty side has no area: its cost is not a number, and no candidate
            if (lc == 0 || lc == n) continue;
            const float cost = __fadd_rn(__fmul_rn(area3(mn, mx), __uint2float_rn(lc)),
                                         __fmul_rn(val[lc * T], __uint2float_rn(n - lc)));
            if (cost < best) best = cost, bax = a, blc = lc, coord = plane;
          }
        }
        if (bax < 0) {
          if (!(parent_cost < 1e34f)) atomicOr(&counters[kError], kErrDegenerate);
          continue;
        }
        if (parent_cost < best) continue;
        uint32_t left = 0;
        for (uint32_t i = 0; i < n; i++) {
          const uint32_t j = nib(cur, b + i);
          const float* q = box + 6 * j * T;
          if (centroid(q[bax * T], q[(3 + bax) * T]) <= coord) left |= 1u << j;
        }
        if (__popc(left) != (int)blc) {
          atomicOr(&counters[kError], kErrPartition);
          continue;
        }
        cur = part_order(cur, b, n, blc, left);
#pragma unroll
        for (int a = 0; a < 3; a++) ord[a] = part_order(ord[a], b, n, blc, left);
        node[k * T] = w | (blc << 9);
        node[(2 * splits + 1) * T] = b | (blc << 4) | ((dep + 1) << 14);
        node[(2 * splits + 2) * T] = (b + blc) | ((n - blc) << 4) | ((dep + 1) << 14);
        splits++;
      }
    }
    // the warp's nodes from the arena with one atomic
    const uint32_t need = 2u * splits;
    uint32_t inc = need;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += y;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&counters[kArenaCount], inc);
    base = __shfl_sync(0xffffffffu, base, 31) + inc - need;
    if (base + need > cap) {
      if (need) atomicOr(&counters[kError], kErrArena);
      continue;
    }
    uint32_t made = 0;
    for (uint32_t k = 0; in && k <= 2 * splits; k++) {
      const uint32_t w = node[k * T], b = w & 15u, n = (w >> 4) & 31u, lc = (w >> 9) & 31u, dep = w >> 14;
      if (lc == 0) continue;
      const int32_t ni = k == 0 ? root : (int32_t)(base + k - 1);
      const uint32_t cid = base + 2 * made++;
      for (uint32_t side = 0; side < 2; side++) {
        const uint32_t cb = side ? b + lc : b, cn = side ? n - lc : lc;
        float mn[3] = {1e34f, 1e34f, 1e34f}, mx[3] = {-1e34f, -1e34f, -1e34f};
        for (uint32_t i = 0; i < cn; i++) {
          const float* q = box + 6 * nib(cur, cb + i) * T;
          for (int c = 0; c < 3; c++) mn[c] = fminf(mn[c], q[c * T]), mx[c] = fmaxf(mx[c], q[(3 + c) * T]);
        }
        arena[cid + side] = make_node(mn, mx, first + cb, cn, ni, depth0 + (int32_t)dep + 1);
      }
    }
    // after every child record (each written with left = -1)
    made = 0;
    for (uint32_t k = 0; in && k <= 2 * splits; k++)
      if ((node[k * T] >> 9) & 31u) arena[k == 0 ? root : (int32_t)(base + k - 1)].left = (int32_t)(base + 2 * made++);
    if (splits)
      for (uint32_t i = 0; i < count; i++) prims[first + i] = id[nib(cur, i) * T];
  }
}

// ---------------------------------------------------------------- collapse
__device__ __forceinline__ bool is_quad(const BNode& b) { return b.left >= 0 && (b.depth & 1) == 0; }

__global__ void k_qcount(BNode* arena, uint32_t* arrive, const uint32_t* counters_ro, uint32_t* counters) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool leaf = i < counters_ro[kArenaCount] && arena[i].left < 0;
  const uint32_t most = __reduce_max_sync(0xffffffffu, leaf ? (uint32_t)arena[i].count : 0u);
  if ((threadIdx.x & 31) == 0 && most > __ldcg(&counters[kMaxLeaf])) atomicMax(&counters[kMaxLeaf], most);
  if (!leaf) return;
  int32_t cur = (int32_t)i;
  while (true) {
    const int32_t p = arena[cur].parent;
    if (p < 0) break;
    __threadfence();
    if (atomicAdd(&arrive[p], 1u) == 0) return;  // the sibling's subtree is not finished yet
    __threadfence();
    const int32_t l = arena[p].left;
    const uint32_t q = __ldcg(&arena[l].qcount) + __ldcg(&arena[l + 1].qcount) + ((arena[p].depth & 1) == 0 ? 1u : 0u);
    __stcg(&arena[p].qcount, q);
    cur = p;
  }
}

__global__ void k_qindex(const BNode* __restrict__ arena, const uint32_t* counters_ro, uint32_t* qidx,
                         uint32_t* counters) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool quad = i < counters_ro[kArenaCount] && is_quad(arena[i]);
  const uint32_t deep = __reduce_max_sync(0xffffffffu, quad ? (uint32_t)(arena[i].depth / 2 + 1) : 0u);
  if ((threadIdx.x & 31) == 0 && deep > __ldcg(&counters[kQuadDepth])) atomicMax(&counters[kQuadDepth], deep);
  if (!quad) return;
  // pre-order position: one for each quad ancestor step, plus the quad nodes of
  // every earlier slot (MergeNodes visits slots left to right, depth first)
  uint32_t idx = 0;
  int32_t cur = (int32_t)i;
  while (cur != 0) {
    const int32_t y = arena[cur].parent, p = arena[y].parent;
    const int32_t ly = arena[y].left, lp = arena[p].left;
    idx += 1;
    if (cur == ly + 1) idx += arena[ly].qcount;
    if (y == lp + 1) idx += arena[lp].qcount;
    cur = p;
  }
  qidx[i] = idx;
}

__device__ __forceinline__ void set_slot(QuadNode& q, int s, const float mn[3], const float mx[3], int32_t child,
                                         int32_t count) {
  q.bminx[s] = mn[0], q.bminy[s] = mn[1], q.bminz[s] = mn[2];
  q.bmaxx[s] = mx[0], q.bmaxy[s] = mx[1], q.bmaxz[s] = mx[2];
  q.childs[s] = child;
  q.counts[s] = count;
}

__global__ void k_qwrite(const BNode* __restrict__ arena, const uint32_t* counters_ro, const uint32_t* __restrict__ qidx,
                         uint32_t nq, QuadNode* quad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= counters_ro[kArenaCount]) return;
  const BNode b = arena[i];
  const float big[3] = {1e34f, 1e34f, 1e34f}, nbig[3] = {-1e34f, -1e34f, -1e34f};
  QuadNode q;
  int num = 0;
  if (i == 0 && b.left < 0) {
    // a root that is a leaf becomes child 0 of the quad root (the reference
    // would leave the tree empty, src/BVH/MBVHNode.cu:233-237)
    set_slot(q, num++, b.mn, b.mx, b.first, b.count);
  } else {
    if (!is_quad(b)) return;
    auto slot = [&](int32_t s) {
      const BNode& c = arena[s];
      if (c.left < 0) set_slot(q, num++, c.mn, c.mx, c.first, c.count);
      else set_slot(q, num++, c.mn, c.mx, (int32_t)qidx[s], -1);
    };
    for (int side = 0; side < 2; side++) {
      const int32_t ci = b.left + side;
      const BNode& c = arena[ci];
      if (c.left < 0) {
        set_slot(q, num++, c.mn, c.mx, c.first, c.count);
      } else {
        slot(c.left);
        slot(c.left + 1);
      }
    }
  }
  for (int s = num; s < 4; s++) set_slot(q, s, big, nbig, -1, 0);
  const uint32_t at_idx = i == 0 ? 0u : qidx[i];
  if (at_idx < nq) quad[at_idx] = q;
}

// Turns quad nodes into traversal nodes where they lie: the planes are the same, the
// references take the place of childs and counts.
__global__ void k_qdev(QNodeDev* nodes, uint32_t nq, uint32_t shift) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const int4 ch = nodes[i].child, cnt = nodes[i].meta;  // QuadNode: childs, counts
  auto ref = [&](int32_t count, int32_t child) {
    return count == -1 ? child
                       : (count > 0 ? (int32_t)(0x80000000u | ((uint32_t)count << shift) | (uint32_t)child) : kEmptyChild);
  };
  nodes[i].child = make_int4(ref(cnt.x, ch.x), ref(cnt.y, ch.y), ref(cnt.z, ch.z), ref(cnt.w, ch.w));
  nodes[i].meta = make_int4(0, 0, 0, 0);
}

__global__ void k_tris(const float4* __restrict__ v, const uint4* __restrict__ idx, const uint32_t* __restrict__ prims,
                       uint32_t n, float4* tris) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t p = prims[j];
  const uint4 t = idx[p];
  const float4 a = v[t.x], b = v[t.y], c = v[t.z];
  const float4 q0 = make_float4(a.x, a.y, a.z, __uint_as_float(p));
  const float2 q1 = make_float2(__fsub_rn(b.x, a.x), __fsub_rn(b.y, a.y));
  float4* o = tris + kTriFloat4 * (size_t)j;
  o[0] = q0;
  *reinterpret_cast<float2*>(o + 1) = q1;
  o[2] = make_float4(__fsub_rn(b.z, a.z), __fsub_rn(c.x, a.x), __fsub_rn(c.y, a.y), __fsub_rn(c.z, a.z));
  if (j == 0) return;
  o -= kTriFloat4;  // the part of this triangle that the one before it carries
  reinterpret_cast<float2*>(o + 1)[1] = q1;
  o[3] = q0;
}

unsigned blocks(uint64_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

#define GB_TRY(call)                      \
  do {                                    \
    cudaError_t e_ = (call);              \
    if (e_ != cudaSuccess) return e_;     \
  } while (0)

}  // namespace

size_t gpu_bvh_scratch_bytes(uint32_t n) { return Layout(n).total; }

cudaError_t gpu_bvh_build(const DevScene& sc, void* scratch, uint32_t* host_counters, cudaStream_t s,
                          GpuBvhResult& r) {
  const uint32_t n = sc.tri_count;
  const Layout L(n);
  uint32_t* counters = at<uint32_t>(scratch, L.counters);
  PrimBox* box = at<PrimBox>(scratch, L.box);
  uint32_t* prims = at<uint32_t>(scratch, L.prims);
  uint32_t* tmp = at<uint32_t>(scratch, L.tmp);
  BNode* arena = at<BNode>(scratch, L.arena);
  uint32_t* arrive = at<uint32_t>(scratch, L.arrive);
  uint32_t* qidx = at<uint32_t>(scratch, L.qidx);

  // the levels' second buffer and partition bits lie where the quad phase works later
  LevelArgs A;
  A.arena = arena;
  A.large[0] = at<int32_t>(scratch, L.large0), A.large[1] = at<int32_t>(scratch, L.large1);
  A.max_large = L.max_large;
  A.mid = at<int32_t>(scratch, L.mid);
  A.max_mid = L.max_mid, A.mid_most = L.mid_most;
  A.small = at<int32_t>(scratch, L.small);
  A.counters = counters;
  A.cap = L.cap;
  A.chunk = L.chunk, A.max_chunks = L.max_chunks;
  A.chunks = at<Chunk>(scratch, L.chunks);
  A.split = at<Split>(scratch, L.split);
  A.bins = at<uint32_t>(scratch, L.bins);
  A.chunk_left = at<uint32_t>(scratch, L.chunk_left);
  A.left = arrive;
  A.box = box;
  A.buf[0] = tmp, A.buf[1] = qidx;
  A.prims = prims;

  k_init<<<1, 32, 0, s>>>(counters);
  k_prep<<<blocks(n, 256), 256, 0, s>>>(sc.verts, sc.idx, n, box, n > L.mid_most ? A.buf[0] : prims, counters);
  k_root<<<1, 1, 0, s>>>(arena, A.large[0], A.mid, A.small, n, L.mid_most, counters);
  GB_TRY(cudaGetLastError());
  GB_TRY(cudaMemcpyAsync(host_counters, counters, 4 * kCounterWords, cudaMemcpyDeviceToHost, s));
  GB_TRY(cudaStreamSynchronize(s));
  uint64_t nl = host_counters[kLarge];
  int par = 0;
  // Up to four levels are issued before the counters are read back (12 us each time),
  // while all their nodes could be large ones: a level that turns out empty costs
  // five launches.
  while (nl > 0) {
    if (nl > L.max_large) return cudaErrorInvalidValue;
    int batch = 1;
    while (batch < 4 && (nl << batch) * L.mid_most <= n) batch++;
    for (int i = 0; i < batch; i++, par ^= 1) {
      const uint64_t most = std::min<uint64_t>(nl << i, L.max_large);
      const unsigned gn = blocks(most * 32, 256);
      const unsigned gc = (unsigned)std::min<uint64_t>((uint64_t)n / L.chunk + most + 1, L.max_chunks);
      GB_TRY(launch_after(k_chunks, gn, 256, 0, s, A, par));
      GB_TRY(launch_after(k_bin, gc, 256, 0, s, A, par));
      GB_TRY(launch_after(k_split, gn, 256, 0, s, A, par));
      GB_TRY(launch_after(k_part_count, gc, 256, 0, s, A, par));
      GB_TRY(launch_after(k_part_scatter, gc, 256, 0, s, A, par));
    }
    GB_TRY(cudaGetLastError());
    GB_TRY(cudaMemcpyAsync(host_counters, counters, 4 * kCounterWords, cudaMemcpyDeviceToHost, s));
    GB_TRY(cudaStreamSynchronize(s));
    nl = host_counters[kLarge + par];
    if (host_counters[kError]) break;
  }
  if (host_counters[kMid] > 0 && !host_counters[kError]) {
    const unsigned threads = n > kFewMid ? 256 : 512;
    auto kernel = L.mid_most == 1024 ? k_mid<1024, 256> : n > kFewMid ? k_mid<2048, 256> : k_mid<2048, 512>;
    const size_t shared = kMidBytes * L.mid_most;
    GB_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared));
    GB_TRY(launch_after(kernel, std::min(host_counters[kMid], L.max_mid), threads, shared, s, A));
  }
  if (n >= 4 && !host_counters[kError]) {
    // how many subtrees the warps have is known on the device
    const int sms = sm_count();
    const unsigned g = (unsigned)std::min<uint64_t>(blocks((uint64_t)n / 4, kSmallWarps), (uint64_t)sms * 8);
    GB_TRY(cudaMemsetAsync(counters + kTasks, 0, 4, s));
    // the levels' first buffer (4 bytes per primitive) is free now: it takes the tasks
    k_small<<<g, kSmallWarps * 32, 0, s>>>(arena, A.small, counters, box, prims, counters, L.cap, tmp);
    GB_TRY(cudaGetLastError());
    GB_TRY(cudaFuncSetAttribute(k_leaf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLeafShared));
    int per_sm = 0;
    GB_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_leaf, kLeafThreads, kLeafShared));
    const unsigned gl = (unsigned)std::min<uint64_t>(blocks((uint64_t)n / 4 + 1, kLeafThreads / 32),
                                                     (uint64_t)sms * std::max(1, per_sm));
    k_leaf<<<gl, kLeafThreads, kLeafShared, s>>>(arena, tmp, box, prims, counters, L.cap);
    GB_TRY(cudaGetLastError());
  }
  GB_TRY(cudaMemsetAsync(arrive, 0, 4 * (size_t)L.cap, s));
  // arena size bound for the grids below: the count is read on the device
  GB_TRY(cudaMemcpyAsync(host_counters, counters, 4 * kCounterWords, cudaMemcpyDeviceToHost, s));
  GB_TRY(cudaStreamSynchronize(s));
  const uint32_t nb = host_counters[kArenaCount];
  k_qcount<<<blocks(nb, 256), 256, 0, s>>>(arena, arrive, counters, counters);
  k_qindex<<<blocks(nb, 256), 256, 0, s>>>(arena, counters, qidx, counters);
  GB_TRY(cudaGetLastError());
  BNode root;
  GB_TRY(cudaMemcpyAsync(host_counters, counters, 4 * kCounterWords, cudaMemcpyDeviceToHost, s));
  GB_TRY(cudaMemcpyAsync(&root, arena, sizeof(BNode), cudaMemcpyDeviceToHost, s));
  GB_TRY(cudaStreamSynchronize(s));
  r.binary_nodes = host_counters[kArenaCount];
  r.error = host_counters[kError];
  r.max_leaf = host_counters[kMaxLeaf];
  if (root.left < 0) {
    r.quad_nodes = 1;
    r.depth = 1;
  } else {
    r.quad_nodes = root.qcount;
    r.depth = host_counters[kQuadDepth];
  }
  return cudaSuccess;
}

cudaError_t launch_quad_to_dev(QNodeDev* nodes, uint32_t nq, uint32_t leaf_shift, cudaStream_t s) {
  if (nq) k_qdev<<<blocks(nq, 256), 256, 0, s>>>(nodes, nq, leaf_shift);
  return cudaGetLastError();
}

cudaError_t launch_leaf_tris(const DevScene& sc, const uint32_t* prims, uint32_t n, float4* tris, cudaStream_t s) {
  if (n) k_tris<<<blocks(n, 256), 256, 0, s>>>(sc.verts, sc.idx, prims, n, tris);
  return cudaGetLastError();
}

cudaError_t gpu_bvh_emit(const DevScene& sc, void* scratch, const GpuBvhResult& r, uint32_t leaf_shift, QNodeDev* nodes,
                         float4* tris, uint32_t* prims_out, cudaStream_t s) {
  const uint32_t n = sc.tri_count;
  const Layout L(n);
  const uint32_t* counters = at<uint32_t>(scratch, L.counters);
  const BNode* arena = at<BNode>(scratch, L.arena);
  const uint32_t* qidx = at<uint32_t>(scratch, L.qidx);
  const uint32_t* prims = at<uint32_t>(scratch, L.prims);
  k_qwrite<<<blocks(r.binary_nodes, 256), 256, 0, s>>>(arena, counters, qidx, r.quad_nodes,
                                                       reinterpret_cast<QuadNode*>(nodes));
  k_qdev<<<blocks(r.quad_nodes, 256), 256, 0, s>>>(nodes, r.quad_nodes, leaf_shift);
  k_tris<<<blocks(n, 256), 256, 0, s>>>(sc.verts, sc.idx, prims, n, tris);
  GB_TRY(cudaGetLastError());
  GB_TRY(cudaMemcpyAsync(prims_out, prims, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
  return cudaSuccess;
}


// ================================================================ 8-wide quantised collapse
namespace {

enum WCounter : int {
  kWidePrims = 0,
  kWideError = 1,
  kWideLevel = 2,                         // the nodes of each level (from the second on)
  kWideLevels = 64,
  kWideFirst = kWideLevel + kWideLevels,  // and the first one's index
  kWideCounterWords = kWideFirst + kWideLevels
};
enum : uint32_t { kWErrSlots = 1, kWErrCapacity = 2, kWErrQuant = 4 };

struct WLayout {
  size_t nodes, list0, list1, counters, total;
  uint32_t cap;
  explicit WLayout(uint32_t binary_nodes) {
    cap = binary_nodes / 2 + 2;  // inner binary nodes + the root
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t a = o;
      o += (bytes + 255) & ~(size_t)255;
      return a;
    };
    nodes = take(sizeof(WNode8) * (size_t)cap);
    list0 = take(sizeof(uint32_t) * (size_t)cap);
    list1 = take(sizeof(uint32_t) * (size_t)cap);
    counters = take(4 * kWideCounterWords);
    total = o;
  }
};

__device__ __forceinline__ uint32_t leaf_slots(int32_t count) { return count <= 0 ? 1u : (uint32_t)(count + 2) / 3u; }
__device__ __forceinline__ float pow2(int biased) { return __int_as_float(biased << 23); }

// Smallest biased exponent whose 255 steps from p reach hi (fma as the traversal evaluates it).
__device__ __forceinline__ int quant_exponent(float p, float hi) {
  const float ext = __fsub_rn(hi, p);
  int e = 1;
  if (ext > 0.0f) {
    int k = 0;
    frexpf(__fdiv_rn(ext, 255.0f), &k);
    e = max(1, min(254, k + 127));
  }
  while (e < 254 && __fmaf_rn(pow2(e), 255.0f, p) < hi) e++;
  return e;
}

// Outward 8-bit bounds of [lo, hi] on the grid p + s*q; false if none fits.
__device__ __forceinline__ bool quantise(float p, float s, float lo, float hi, uint8_t& qlo, uint8_t& qhi) {
  float fl = floorf(__fdiv_rn(__fsub_rn(lo, p), s)), fh = ceilf(__fdiv_rn(__fsub_rn(hi, p), s));
  int ql = (int)fminf(fmaxf(fl, 0.0f), 255.0f), qh = (int)fminf(fmaxf(fh, 0.0f), 255.0f);
  while (ql > 0 && __fmaf_rn(s, (float)ql, p) > lo) ql--;
  while (qh < 255 && __fmaf_rn(s, (float)qh, p) < hi) qh++;
  qlo = (uint8_t)ql, qhi = (uint8_t)qh;
  return __fmaf_rn(s, (float)ql, p) <= lo && __fmaf_rn(s, (float)qh, p) >= hi;
}

__device__ __forceinline__ uint32_t wsplit(const WideCost& c, int i) { return (c.split >> (3 * (i - 2))) & 7u; }

// The binary nodes that become the entries of wide node b (at most eight), left to
// right; leafy[k]: entry k becomes leaf slots (its primitive range, three per slot).
// Returns their number, -1 when they don't fit.
__device__ __forceinline__ int wide_entries(const BNode* arena, const WideCost* cost, uint32_t bin, const BNode& b,
                                            int32_t F[8], bool leafy[8]) {
  int nf = 0;
  if (b.left < 0) {
    F[nf] = (int32_t)bin, leafy[nf++] = true;
  } else {
    // the slots of least cost (the optimal n-wide collapse of Ylitie, Karras and
    // Laine, HPG 2017): k of 8 to the left child, then each side as its table says
    const int32_t L = b.left, R = L + 1;
    float best = 3e38f;
    int bk = 1;
    for (int k = 1; k < 8; k++) {
      const float c = __fadd_rn(cost[L].c[k - 1], cost[R].c[8 - k - 1]);
      if (c < best) best = c, bk = k;
    }
    int32_t stn[16];
    int sti[16];
    int sp = 0;
    stn[sp] = R, sti[sp++] = 8 - bk;
    stn[sp] = L, sti[sp++] = bk;
    while (sp > 0) {
      const int32_t x = stn[--sp];
      int ix = sti[sp];
      const BNode& c = arena[x];
      while (ix > 1 && (c.left < 0 || wsplit(cost[x], ix) == 0)) ix--;
      if (ix == 1) {
        if (nf >= 8) return -1;
        F[nf] = x, leafy[nf++] = c.left < 0 || cost[x].leaf1 != 0;
        continue;
      }
      const int k = (int)wsplit(cost[x], ix);
      if (sp + 2 > 16) return -1;
      stn[sp] = c.left + 1, sti[sp++] = ix - k;
      stn[sp] = c.left, sti[sp++] = k;
    }
  }
  uint32_t used = 0;
  for (int k = 0; k < nf; k++) used += leafy[k] ? leaf_slots(arena[F[k]].count) : 1u;
  return used > 8 ? -1 : nf;
}

// One level: its nodes follow the previous level's. Children and triangles are
// placed for a warp's nodes at once (three atomics a node on shared counters: 536
// against 500 us for the levels of a 1 M-triangle tree).
__global__ void __launch_bounds__(128) k_wcollapse(const BNode* __restrict__ arena, const uint32_t* __restrict__ bprims,
                                                   const WideCost* __restrict__ cost, const float4* __restrict__ v,
                                                   const uint4* __restrict__ idx, const uint32_t* in, int level,
                                                   uint32_t* out, uint32_t* counters, WNode8* wn, float4* wtris,
                                                   uint32_t cap, uint32_t n_prims) {
  after_previous();
  if (counters[kWideError]) return;  // an earlier level failed: its list has gaps
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t first = level ? counters[kWideFirst + level] : 0u, n_in = level ? counters[kWideLevel + level] : 1u;
  if (i == 0) counters[kWideFirst + level + 1] = first + n_in;
  if ((i & ~31u) >= n_in) return;  // whole warp
  const bool live = i < n_in;
  int32_t F[8];
  bool leafy[8];
  int nf = 0;
  uint32_t n_int = 0, n_tri = 0;
  BNode b;
  if (live) {
    const uint32_t bin = level ? in[i] : 0u;
    b = arena[bin];
    nf = wide_entries(arena, cost, bin, b, F, leafy);
    if (nf < 0) atomicOr(&counters[kWideError], kWErrSlots);
    for (int k = 0; k < nf; k++) {
      if (!leafy[k]) n_int++;
      else n_tri += (uint32_t)arena[F[k]].count;
    }
  }
  const uint32_t out_base = warp_alloc(&counters[kWideLevel + level + 1], n_int);
  const uint32_t prim_base = warp_alloc(&counters[kWidePrims], n_tri);
  const uint32_t child_base = first + n_in + out_base;
  if (!live || nf < 0) return;
  if (child_base + n_int > cap || prim_base + n_tri > n_prims) {
    atomicOr(&counters[kWideError], kWErrCapacity);
    return;
  }
  WNode8 w;
  memset(&w, 0, sizeof(w));
  const float p[3] = {b.mn[0], b.mn[1], b.mn[2]};
  float sc[3];
  for (int a = 0; a < 3; a++) {
    const int e = quant_exponent(p[a], b.mx[a]);
    w.e[a] = (uint8_t)e;
    sc[a] = pow2(e);
  }
  w.px = p[0], w.py = p[1], w.pz = p[2];
  w.child_base = n_int ? child_base : 0u;
  w.prim_base = n_tri ? prim_base : 0u;
  bool ok = true;
  int slot = 0;
  uint32_t rank = 0, off = 0;
  for (int k = 0; k < nf; k++) {
    const BNode& c = arena[F[k]];
    if (!leafy[k]) {
      for (int a = 0; a < 3; a++) ok &= quantise(p[a], sc[a], c.mn[a], c.mx[a], w.qlo[a][slot], w.qhi[a][slot]);
      w.meta[slot] = (uint8_t)(0x80u | rank);
      w.imask |= (uint8_t)(1u << slot);
      out[out_base + rank] = (uint32_t)F[k];
      rank++, slot++;
      continue;
    }
    for (int32_t j = 0; j < c.count; j += 3) {
      const int cnt = min(3, c.count - j);
      float mn[3] = {1e34f, 1e34f, 1e34f}, mx[3] = {-1e34f, -1e34f, -1e34f};
      for (int t = 0; t < cnt; t++) {
        const uint32_t prim = bprims[c.first + j + t];
        const uint4 ti = idx[prim];
        const float4 a = v[ti.x], bb = v[ti.y], cc = v[ti.z];
        mn[0] = fminf(mn[0], fminf(a.x, fminf(bb.x, cc.x))), mx[0] = fmaxf(mx[0], fmaxf(a.x, fmaxf(bb.x, cc.x)));
        mn[1] = fminf(mn[1], fminf(a.y, fminf(bb.y, cc.y))), mx[1] = fmaxf(mx[1], fmaxf(a.y, fmaxf(bb.y, cc.y)));
        mn[2] = fminf(mn[2], fminf(a.z, fminf(bb.z, cc.z))), mx[2] = fmaxf(mx[2], fmaxf(a.z, fmaxf(bb.z, cc.z)));
        float4* o = wtris + 3 * (size_t)(prim_base + off + t);
        o[0] = make_float4(a.x, a.y, a.z, __uint_as_float(prim));
        o[1] = make_float4(bb.x, bb.y, bb.z, 0.0f);
        o[2] = make_float4(cc.x, cc.y, cc.z, 0.0f);
      }
      for (int a = 0; a < 3; a++) ok &= quantise(p[a], sc[a], mn[a], mx[a], w.qlo[a][slot], w.qhi[a][slot]);
      w.meta[slot] = (uint8_t)(((uint32_t)cnt << 5) | off);
      off += (uint32_t)cnt;
      slot++;
    }
  }
  if (!ok) atomicOr(&counters[kWideError], kWErrQuant);
  wn[first + i] = w;
}

}  // namespace

size_t gpu_wbvh_scratch_bytes(uint32_t binary_nodes) { return WLayout(binary_nodes).total; }

cudaError_t gpu_wbvh_collapse(const DevScene& sc, const void* arena_v, const uint32_t* bprims, const WideCost* cost,
                              void* scratch2, uint32_t binary_nodes, float4* tris, uint32_t* host_counters,
                              cudaStream_t s, uint32_t* wide_nodes, uint32_t* depth, uint32_t* error) {
  const uint32_t n = sc.tri_count;
  const WLayout W(binary_nodes);
  // both binary builders write this 48-byte node layout (BNode here, FNodeD in bvh_gpu_fast.cu)
  const BNode* arena = static_cast<const BNode*>(arena_v);
  WNode8* wn = at<WNode8>(scratch2, W.nodes);
  uint32_t* lists[2] = {at<uint32_t>(scratch2, W.list0), at<uint32_t>(scratch2, W.list1)};
  uint32_t* counters = at<uint32_t>(scratch2, W.counters);
  GB_TRY(cudaMemsetAsync(counters, 0, 4 * kWideCounterWords, s));
  // four levels per readback, as the quad tree's (a node has at most eight children)
  uint32_t n_in = 1, levels = 0, nodes = 0;
  while (n_in > 0) {
    const int batch = std::min(4, kWideLevels - 1 - (int)levels);
    if (batch <= 0) {
      *error = kWErrCapacity;
      return cudaSuccess;
    }
    for (int i = 0; i < batch; i++) {
      const int l = (int)levels + i;
      const uint64_t most = std::min<uint64_t>((uint64_t)n_in << (3 * i), W.cap);
      GB_TRY(launch_after(k_wcollapse, blocks(most, 128), 128, 0, s, arena, bprims, cost, sc.verts, sc.idx, lists[l & 1], l,
                          lists[(l + 1) & 1], counters, wn, tris, W.cap, n));
    }
    GB_TRY(cudaMemcpyAsync(host_counters, counters, 4 * kWideLevel, cudaMemcpyDeviceToHost, s));
    GB_TRY(cudaMemcpyAsync(host_counters + kWideLevel, counters + kWideLevel + levels + 1, 4 * (size_t)batch,
                           cudaMemcpyDeviceToHost, s));
    GB_TRY(cudaStreamSynchronize(s));
    for (int i = 0; i < batch && n_in > 0; i++) nodes += n_in, n_in = host_counters[kWideLevel + i], levels++;
    if (host_counters[kWideError]) break;
  }
  *wide_nodes = nodes;
  *depth = levels;
  *error = host_counters[kWideError] | (host_counters[kWidePrims] != n ? kWErrCapacity : 0u);
  return cudaSuccess;
}

namespace {
__global__ void __launch_bounds__(256) k_wdev(const WNode8* __restrict__ in, uint32_t n, WNodeDev* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const WNode8 w = in[i];
  WNodeDev d;
  d.p[0] = w.px, d.p[1] = w.py, d.p[2] = w.pz;
  d.imask = w.imask;
  for (int a = 0; a < 3; a++) {
    d.e[a] = w.e[a];
    for (int k = 0; k < 8; k++) d.q[a][0][k] = w.qlo[a][k], d.q[a][1][k] = w.qhi[a][k];
  }
  for (int k = 0; k < 8; k++) {
    const uint32_t m = w.meta[k];
    d.ent[k] = m == 0 ? 0u
               : (m & 0x80u) ? w.child_base + (m & 7u)
                             : (0x80000000u | ((m >> 5) << 29) | (w.prim_base + (m & 31u)));
  }
  out[i] = d;
}
}  // namespace

cudaError_t gpu_wbvh_copy_nodes(void* scratch2, uint32_t binary_nodes, WNodeDev* out, uint32_t count, cudaStream_t s) {
  const WLayout W(binary_nodes);
  if (count) k_wdev<<<blocks(count, 256), 256, 0, s>>>(at<WNode8>(scratch2, W.nodes), count, out);
  return cudaGetLastError();
}

namespace {
// The QuadNode a QNodeDev was made from: the planes are the same, childs and counts
// take the place of the references.
struct QuadOut {
  using In = QNodeDev;
  using Out = QuadNode;
  uint32_t shift, first_mask, count_mask;
  __host__ __device__ QuadNode operator()(const QNodeDev& d) const {
    static_assert(sizeof(QuadNode) == sizeof(QNodeDev) && offsetof(QuadNode, childs) == offsetof(QNodeDev, child) &&
                      offsetof(QuadNode, bmaxz) == offsetof(QNodeDev, bmaxz),
                  "same planes");
    QuadNode q;
    memcpy(&q, &d, sizeof(q));
    for (int c = 0; c < 4; c++) {
      const int32_t ref = q.childs[c];
      if (ref == kEmptyChild) q.counts[c] = 0;  // childs -1 as well
      else if (ref >= 0) q.counts[c] = -1;
      else q.counts[c] = (int32_t)(((uint32_t)ref >> shift) & count_mask), q.childs[c] = ref & (int32_t)first_mask;
    }
    return q;
  }
};

// The 80-byte node a WNodeDev was made from.
struct WideOut {
  using In = WNodeDev;
  using Out = WNode8;
  __host__ __device__ WNode8 operator()(const WNodeDev& d) const {
    WNode8 w;
    memset(&w, 0, sizeof(w));
    w.px = d.p[0], w.py = d.p[1], w.pz = d.p[2];
    w.imask = d.imask;
    for (int a = 0; a < 3; a++) {
      w.e[a] = d.e[a];
      for (int k = 0; k < 8; k++) w.qlo[a][k] = d.q[a][0][k], w.qhi[a][k] = d.q[a][1][k];
    }
    // children and triangles are numbered in slot order from the node's first ones
    bool child = false, prim = false;
    for (int k = 0; k < 8; k++) {
      const uint32_t ent = d.ent[k];
      if (ent == 0) continue;
      if (ent & 0x80000000u) {
        const uint32_t first = ent & 0x1fffffffu;
        if (!prim) w.prim_base = first, prim = true;
        w.meta[k] = (uint8_t)((((ent >> 29) & 3u) << 5) | (first - w.prim_base));
      } else {
        if (!child) w.child_base = ent, child = true;
        w.meta[k] = (uint8_t)(0x80u | (ent - w.child_base));
      }
    }
    return w;
  }
};

template <class F>
__global__ void __launch_bounds__(256) k_export(F f, const typename F::In* __restrict__ in, uint32_t n,
                                                typename F::Out* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = f(in[i]);
}

template <class F>
cudaError_t export_nodes(F f, const typename F::In* nodes, uint32_t n, void* to, void* tmp, cudaStream_t s) {
  using In = typename F::In;
  using Out = typename F::Out;
  std::unique_ptr<In[]> host(tmp ? nullptr : new (std::nothrow) In[std::min(n, kExportPiece)]);
  if (!tmp && !host) return cudaErrorMemoryAllocation;
  for (uint32_t i = 0; i < n; i += kExportPiece) {
    const uint32_t c = std::min(n - i, kExportPiece);
    char* dst = (char*)to + (size_t)i * sizeof(Out);
    if (tmp) {
      k_export<F><<<blocks(c, 256), 256, 0, s>>>(f, nodes + i, c, (Out*)tmp);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    cudaError_t e = tmp ? cudaMemcpyAsync(dst, tmp, c * sizeof(Out), cudaMemcpyDeviceToHost, s)
                        : cudaMemcpyAsync(host.get(), nodes + i, c * sizeof(In), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && !tmp) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    for (uint32_t j = 0; !tmp && j < c; j++) {
      const Out o = f(host[j]);
      std::memcpy(dst + j * sizeof(Out), &o, sizeof(Out));  // at any alignment
    }
  }
  return cudaStreamSynchronize(s);
}
}  // namespace

cudaError_t export_quads(const DevBVH& b, void* to, void* tmp, cudaStream_t s) {
  return export_nodes(QuadOut{b.leaf_shift, b.first_mask, b.count_mask}, b.nodes, b.node_count, to, tmp, s);
}
cudaError_t export_wides(const DevWBVH& b, void* to, void* tmp, cudaStream_t s) {
  return export_nodes(WideOut{}, b.nodes, b.node_count, to, tmp, s);
}
}  // namespace ct

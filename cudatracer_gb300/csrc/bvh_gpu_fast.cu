// Device build of the traversal-speed quad tree (ct_bvh_build_fast_device).
//
// The rules of the host builder (bvh_fast.cpp: triangle boxes padded relative
// to their coordinates, 16 centroid bins per axis, the exact sweep for ranges
// of at most 16 primitives, split to one primitive per leaf, the cost-optimal
// four-wide collapse, slots in descending box area), evaluated with the same
// IEEE operations in the same order (__fadd_rn/__fmul_rn/__fdiv_rn: nothing
// is contracted). Box unions are min/max, which is exact and, with no negative
// zero in any box, independent of the order; every partition is stable, as on
// the host. So the quad nodes and the primitive order equal
// ct_bvh_build_fast's byte for byte.
//
// Phases:
//   prep      the largest coordinate magnitude M, padded boxes and centroids,
//             the root box
//   levels    nodes of more than mid_size(n) primitives, level by level: per chunk
//             of primitives the bins (shared memory, flushed into the node's global
//             bins); one warp per node evaluates the 45 bin splits; a bit per
//             primitive and chunk counts give the stable partition into the other
//             level's buffer, and the children's centroid bounds with it
//   mid       one block splits each node down to ranges of at most kWarpMax in
//             shared memory
//   small     one warp splits each subtree of at most kWarpMax primitives by bins
//             down to ranges of at most 16
//   leaf      one thread builds the whole subtree of each such range (the exact
//             sweep), 32 of them per warp
//   cost      the collapse's cost table C(n, 1..4), bottom-up: the second of
//             two sibling subtrees to finish computes the parent
//   collapse  quad nodes level by level from the root, each choosing its slots
//             from the cost table. The host numbers the children of a quad node
//             when it visits that node, visiting in pre-order: so a node's
//             children are numbered from 1 + the number of children of all
//             nodes before it in pre-order (subtree sizes bottom-up, pre-order
//             ranks top-down, an exclusive scan in rank order)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "bvh_build.h"
#include "ct_internal.h"
#include "launch.cuh"

namespace ct {
namespace {

constexpr int kBins = 16;
constexpr int kCands = 3 * (kBins - 1);  // 45 split candidates per node
constexpr int kBinFields = 7;            // count, min key x/y/z, max key x/y/z
constexpr int kBinWords = 3 * kBins * kBinFields;
constexpr uint32_t kLeafMax = 4;
constexpr int32_t kDepthLimit = 60;
constexpr float kPad = 1e-5f;
constexpr uint32_t kSweepMax = 16;
constexpr uint32_t kWarpMax = 128;   // subtrees up to this size: one warp
// Nodes up to this size are split by one block down to those (64 KB of shared memory
// leave three blocks of 2,048 on an SM and six of 1,024). Soups with 2,048 and with 1,024,
// ms: 300,000 triangles 1.32 and 1.29, 1.1 M 2.54 and 2.50, 2.0 M 3.87 and 3.79; a terrain
// of 486,000 1.66 and 1.65.
inline uint32_t mid_size(uint32_t n) { return n > 400000 ? 1024 : 2048; }
// Builds of at most this many triangles leave an SM about one such block, which has 512
// threads then instead of 256. Terrains with 256 and with 512 threads, us: 122,000
// triangles 1,216 and 1,202, 231,000 1,354 and 1,335, 421,000 1,598 and 1,583, 602,000
// 1,918 and 1,972.
constexpr uint32_t kFewMid = 250000;
// Primitives per block of the level kernels: the fewest, as a power of two from
// 256, that leave no more blocks than about one wave holds (8 blocks of 256 threads
// on each SM). A 20,480-triangle build has 80 blocks of one pass over
// their threads rather than 10 of eight (k_fbin 18 -> 8 us a level); above 1.2 M
// triangles the 2,048 of one wave stay (fewer bin flushes).
inline uint32_t chunk_size(uint32_t n) {
  uint32_t c = 256;
  while (c < 2048 && n / c > (uint32_t)sm_count() * 8) c *= 2;
  return c;
}
constexpr int kSmallWarps = 4;
constexpr int kSmallStack = 64;  // depth limit 60: at most 61 pending nodes
constexpr int kScanBlock = 1024;

enum : uint32_t { kErrRange = 1, kErrArena = 2, kErrStack = 4, kErrPartition = 8, kErrQuad = 16 };
enum Counter : int {
  kArenaCount = 0,
  kSmallCount = 1,
  kError = 4,
  kMaxLeaf = 5,
  kMag = 6,
  kChunks = 2,       // 2 words: chunks of the even and of the odd level
  kTasks = kChunks,  // ranges for k_fleaf, once the levels are done
  kMid = 7,          // nodes for k_fmid
  kRootKeys = 8,     // 6 words: min x/y/z, max x/y/z
  kLarge = 14,       // 2 words: large nodes of the even and of the odd level
  kCounterWords = 16,
  // after these, for the quad phase: where each level's nodes begin and how many it has
  kQuadLevels = 64,  // the binary depth limit of 60 bounds them
  kQuadFirst = kCounterWords,
  kQuadCount = kQuadFirst + kQuadLevels,
  kAllWords = kQuadCount + kQuadLevels
};

struct __align__(16) FNodeD {
  float mn[3];
  int32_t first;
  float mx[3];
  int32_t count;
  int32_t left;    // -1 for a leaf, else the left child (right = left + 1)
  int32_t parent;  // -1 at the root
  int32_t depth;
  uint32_t pad;
};
static_assert(sizeof(FNodeD) == 48, "FNodeD");

// C(n, i) for i = 1..4 in c[0..3]; meta bit 0: with one slot the subtree is a
// leaf; bits 8(i-1)..: with i slots, the slots given to the left child (0: as
// with i - 1 slots)
struct __align__(16) FCostD {
  float c[4];
  uint32_t meta;
  uint32_t pad[3];
};
static_assert(sizeof(FCostD) == 32, "FCostD");

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
struct FSplit {
  int32_t mode;  // -1 not split yet, 0 partition by bin, 1 halves in the current order, -2 no chunks
  int32_t kid[2];  // the children's slots of the next level, -1 where they have none
  int32_t axis;
  float lo, scale;
  int32_t bsp;  // primitives with bin < bsp go left
  uint32_t lc;
  uint32_t chunk0;
};

// one quad node (index = breadth-first allocation order)
struct QRec {
  int32_t slot[4];  // binary node of each slot, -1 empty
  int32_t kid[4];   // quad record of an inner slot, else -1
  uint32_t leafmask, nk, size, rank;
  uint32_t number, pad[3];
};
static_assert(sizeof(QRec) == 64, "QRec");

struct Layout {
  size_t box, prims, tmp, arena, cost, arrive, large0, large1, mid, small, chunks, chunk_left, split,
      bins, cbk, qlist, qrec, scan, sums, counters, total;
  uint32_t chunk, cap, qcap, mid_most, max_large, max_mid, max_chunks, max_small, max_sums;
  explicit Layout(uint32_t n, int wide = 0) {
    cap = 2 * n + 2;
    qcap = n + 2;
    mid_most = mid_size(n);
    max_large = n / (mid_most + 1) + 2;
    max_mid = n / (kWarpMax + 1) + 2;
    chunk = chunk_size(n);
    max_chunks = n / chunk + max_large + 2;
    max_small = n / 2 + 2;
    max_sums = qcap / kScanBlock + 2;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += (bytes + 255) & ~(size_t)255;
      return at;
    };
    box = take(sizeof(PrimBox) * (size_t)n);
    prims = take(4 * (size_t)n);
    tmp = take(4 * (size_t)n);
    arena = take(sizeof(FNodeD) * (size_t)cap);
    cost = take((wide ? sizeof(WideCost) : sizeof(FCostD)) * (size_t)cap);
    arrive = take(4 * (size_t)cap);
    large0 = take(4 * (size_t)max_large);
    large1 = take(4 * (size_t)max_large);
    mid = take(4 * (size_t)max_mid);
    small = take(4 * (size_t)max_small);
    chunks = take(sizeof(Chunk) * (size_t)max_chunks);
    chunk_left = take(4 * (size_t)max_chunks);
    split = take(sizeof(FSplit) * (size_t)max_large);
    bins = take(4 * (size_t)kBinWords * max_large);
    cbk = take(2 * 4 * 6 * (size_t)max_large);
    qlist = take(4 * (size_t)qcap);
    qrec = take(sizeof(QRec) * (size_t)qcap);
    scan = take(4 * (size_t)qcap);
    sums = take(4 * (size_t)max_sums);
    counters = take(4 * kAllWords);
    total = o;
  }
};

template <typename T>
T* at(void* base, size_t off) {
  return reinterpret_cast<T*>(static_cast<char*>(base) + off);
}

// order-preserving float <-> uint32 keys for atomic and warp min/max
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
// std::min / std::max as the host evaluates them
__device__ __forceinline__ float gmin(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float gmax(float a, float b) { return a < b ? b : a; }
__device__ __forceinline__ float comp(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// the box's centre as k_fprep checked it
__device__ __forceinline__ float4 centre(const PrimBox& b) {
  return make_float4(__fmul_rn(0.5f, __fadd_rn(b.lo.x, b.hi.x)), __fmul_rn(0.5f, __fadd_rn(b.lo.y, b.hi.y)),
                     __fmul_rn(0.5f, __fadd_rn(b.lo.z, b.hi.z)), 0.0f);
}

// farea (bvh_fast.cpp): surface area with extents scaled by s
__device__ __forceinline__ float farea(const float mn[3], const float mx[3], float s) {
  const float dx = __fmul_rn(__fsub_rn(mx[0], mn[0]), s), dy = __fmul_rn(__fsub_rn(mx[1], mn[1]), s),
              dz = __fmul_rn(__fsub_rn(mx[2], mn[2]), s);
  if (dx < 0.0f) return 0.0f;
  return __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx)));
}
// bin_of (bvh_fast.cpp)
__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
  const float f = __fmul_rn(__fsub_rn(c, lo), scale);
  if (!(f >= 1.0f)) return 0;
  if (f >= (float)(kBins - 1)) return kBins - 1;
  return (int)f;
}
// per-axis bin origin and scale from a range's centroid bounds (6 keys)
__device__ __forceinline__ void bin_frame(const uint32_t* k, float lo[3], float scale[3]) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float mn = unkey(k[a]), mx = unkey(k[3 + a]);
    const float ext = __fsub_rn(mx, mn);
    lo[a] = mn;
    scale[a] = ext > 0.0f ? __fdiv_rn((float)kBins, ext) : 0.0f;
  }
}

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
      uint32_t* e = bins + (a * kBins + b0) * kBinFields + lane;
      if (lane == 0) atomicAdd(e, mine);
      else if (lane < 4) atomicMin(e, mine);
      else if (lane < 7) atomicMax(e, mine);
      rem &= ~same;
    }
    if ((rem >> lane) & 1u) {
      uint32_t* e = bins + (a * kBins + bin[a]) * kBinFields;
      atomicAdd(e, 1u);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        atomicMin(e + 1 + k, key[k]);
        atomicMax(e + 4 + k, key[3 + k]);
      }
    }
  }
}

// The bins of one primitive per axis (-1 where all centroids coincide).
__device__ __forceinline__ void bins_of(const float lo[3], const float scale[3], const float4& c, int bin[3]) {
#pragma unroll
  for (int a = 0; a < 3; a++) bin[a] = scale[a] > 0.0f ? bin_of(comp(c, a), lo[a], scale[a]) : -1;
}

struct Cand {
  float cost;
  int32_t j;  // candidate index a * 15 + i - 1; kCands + 32 when none
  uint32_t lc, rc;
  float lmn[3], lmx[3], rmn[3], rmx[3];
};

__device__ __forceinline__ void bcast_cand(Cand& c, int src) {
  c.cost = __shfl_sync(0xffffffffu, c.cost, src);
  c.j = __shfl_sync(0xffffffffu, c.j, src);
  c.lc = __shfl_sync(0xffffffffu, c.lc, src);
  c.rc = __shfl_sync(0xffffffffu, c.rc, src);
  for (int k = 0; k < 3; k++) {
    c.lmn[k] = __shfl_sync(0xffffffffu, c.lmn[k], src);
    c.lmx[k] = __shfl_sync(0xffffffffu, c.lmx[k], src);
    c.rmn[k] = __shfl_sync(0xffffffffu, c.rmn[k], src);
    c.rmx[k] = __shfl_sync(0xffffffffu, c.rmx[k], src);
  }
}

// First lowest cost over the 45 bin splits in axis-major order (the host's
// strict "cost < best" scan); the whole warp returns the winner, j >= kCands
// when no split qualifies.
//
// Half a warp takes an axis: lane k of it is the split behind bin k, and the left
// and right unions of all splits are two scans over the half. (A candidate per lane
// that walks all bins reads 112 words and decodes 96 keys, twice: k_fsmall took 853
// us of a 2.0 M-triangle build so, 507 with the scans, and the k_fsplit of its 21
// levels 380 and 264.) Unions keep the walk's order, earlier bins on the left, so
// that equal bounds give the same bits.
__device__ __forceinline__ void choose_bin_split(const uint32_t* bins, const float scale[3], float s, int lane,
                                                 Cand& best) {
  const unsigned FULL = 0xffffffffu;
  const int k = lane & 15;
  best.j = kCands + 32;
  best.cost = 0.0f;
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const int a = 2 * pass + (lane >> 4);
    Cand c;
    c.j = kCands + 32;
    c.lc = c.rc = 0;
    for (int x = 0; x < 3; x++) c.lmn[x] = c.rmn[x] = 1e34f, c.lmx[x] = c.rmx[x] = -1e34f;
    if (a < 3 && k < kBins - 1) {
      const uint32_t* e = bins + (a * kBins + k) * kBinFields;
      c.lc = e[0], c.rc = e[kBinFields];
      for (int x = 0; x < 3; x++) {
        c.lmn[x] = gmin(c.lmn[x], unkey(e[1 + x])), c.lmx[x] = gmax(c.lmx[x], unkey(e[4 + x]));
        c.rmn[x] = gmin(c.rmn[x], unkey(e[kBinFields + 1 + x])), c.rmx[x] = gmax(c.rmx[x], unkey(e[kBinFields + 4 + x]));
      }
    }
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
      const uint32_t ul = __shfl_up_sync(FULL, c.lc, off, 16), dr = __shfl_down_sync(FULL, c.rc, off, 16);
      const bool up = k >= off, down = k + off < 16;
      if (up) c.lc += ul;
      if (down) c.rc += dr;
#pragma unroll
      for (int x = 0; x < 3; x++) {
        const float umn = __shfl_up_sync(FULL, c.lmn[x], off, 16), umx = __shfl_up_sync(FULL, c.lmx[x], off, 16);
        const float dmn = __shfl_down_sync(FULL, c.rmn[x], off, 16), dmx = __shfl_down_sync(FULL, c.rmx[x], off, 16);
        if (up) c.lmn[x] = gmin(umn, c.lmn[x]), c.lmx[x] = gmax(umx, c.lmx[x]);
        if (down) c.rmn[x] = gmin(c.rmn[x], dmn), c.rmx[x] = gmax(c.rmx[x], dmx);
      }
    }
    if (a < 3 && k < kBins - 1 && scale[a] > 0.0f && c.lc != 0 && c.rc != 0) {
      c.cost = __fadd_rn(__fmul_rn(farea(c.lmn, c.lmx, s), __uint2float_rn(c.lc)),
                         __fmul_rn(farea(c.rmn, c.rmx, s), __uint2float_rn(c.rc)));
      c.j = a * (kBins - 1) + k;
      // the host's running best starts at 3e38
      if (c.cost < 3e38f && (best.j >= kCands || c.cost < best.cost)) best = c;
    }
  }
  float bc = best.cost;
  int bj = best.j;
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    const float oc = __shfl_xor_sync(FULL, bc, off);
    const int oj = __shfl_xor_sync(FULL, bj, off);
    if (oj < kCands && (bj >= kCands || oc < bc || (oc == bc && oj < bj))) bc = oc, bj = oj;
  }
  if (bj >= kCands) {
    best.j = kCands + 32;
    return;
  }
  bcast_cand(best, bj % (kBins - 1) + (bj / (kBins - 1) == 1 ? 16 : 0));
}

// Union of the boxes of prims[b, e) by one warp (order-free).
__device__ __forceinline__ void warp_union(const PrimBox* box, const uint32_t* prims, uint32_t b,
                                           uint32_t e, int lane, float mn[3], float mx[3]) {
  uint32_t kmn[3] = {fkey(1e34f), fkey(1e34f), fkey(1e34f)}, kmx[3] = {fkey(-1e34f), fkey(-1e34f), fkey(-1e34f)};
  for (uint32_t k = b + lane; k < e; k += 32) {
    const PrimBox v = prim_box(box + prims[k]);
    const float4 l = v.lo, h = v.hi;
    kmn[0] = min(kmn[0], fkey(l.x)), kmn[1] = min(kmn[1], fkey(l.y)), kmn[2] = min(kmn[2], fkey(l.z));
    kmx[0] = max(kmx[0], fkey(h.x)), kmx[1] = max(kmx[1], fkey(h.y)), kmx[2] = max(kmx[2], fkey(h.z));
  }
  for (int k = 0; k < 3; k++) {
    mn[k] = unkey(__reduce_min_sync(0xffffffffu, kmn[k]));
    mx[k] = unkey(__reduce_max_sync(0xffffffffu, kmx[k]));
  }
}

__device__ __forceinline__ FNodeD make_node(const float mn[3], const float mx[3], uint32_t first, uint32_t count,
                                            int32_t parent, int32_t depth) {
  FNodeD b;
  for (int k = 0; k < 3; k++) b.mn[k] = mn[k], b.mx[k] = mx[k];
  b.first = (int32_t)first;
  b.count = (int32_t)count;
  b.left = -1;
  b.parent = parent;
  b.depth = depth;
  b.pad = 0;
  return b;
}

// Queue of a child that a block or a warp splits further (the level kernels keep
// theirs, add_children).
__device__ __forceinline__ void queue_child(int32_t id, uint32_t count, int32_t depth, int32_t* mid, uint32_t max_mid,
                                            int32_t* small, uint32_t max_small, uint32_t* counters) {
  if (count <= 1 || depth >= kDepthLimit) return;  // a leaf
  const bool m = count > kWarpMax;
  const uint32_t s = atomicAdd(&counters[m ? kMid : kSmallCount], 1u), most = m ? max_mid : max_small;
  if (s < most) (m ? mid : small)[s] = id;
  else atomicOr(&counters[kError], kErrArena);
}

// ---------------------------------------------------------------- prep
__global__ void k_finit(uint32_t* counters, uint32_t* cbk) {
  const int w = threadIdx.x;
  if (w < 6) cbk[w] = w < 3 ? fkey(1e34f) : fkey(-1e34f);
  if (w < kCounterWords)
    counters[w] = (w >= kRootKeys && w < kRootKeys + 3) ? fkey(1e34f)
                  : (w >= kRootKeys + 3 && w < kRootKeys + 6) ? fkey(-1e34f)
                                                              : 0u;
}

// Root bounds: reduced over the block before the six counters every block shares
// are touched. With one atomic per warp the 2.0 M-triangle prep spent 290 of its
// us on them.
__device__ __forceinline__ void block_root_keys(uint32_t* root, uint32_t kmn[3], uint32_t kmx[3]) {
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
  if (threadIdx.x < 3) atomicMin(&root[threadIdx.x], red[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&root[threadIdx.x], red[threadIdx.x]);
}

__global__ void __launch_bounds__(256) k_fmag(const float4* __restrict__ v, const uint4* __restrict__ idx, uint32_t n,
                                              uint32_t* counters) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  float m = 0.0f;
  if (i < n) {
    const uint4 t = idx[i];
    const float4 p[3] = {v[t.x], v[t.y], v[t.z]};
    for (int k = 0; k < 3; k++) m = gmax(m, gmax(fabsf(p[k].x), gmax(fabsf(p[k].y), fabsf(p[k].z))));
  }
  // non-negative floats order as their bit patterns
  __shared__ uint32_t red;
  if (threadIdx.x == 0) red = 0;
  __syncthreads();
  const uint32_t r = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) atomicMax(&red, r);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&counters[kMag], red);
}

// prims: the buffer of the first level, or the final one when the root is small.
// cbk: the root's centroid bounds.
// rel_pad: kPad for the traversal-speed quad tree, 0 (exact bounds) for the wide tree
__global__ void __launch_bounds__(256) k_fprep(const float4* __restrict__ v, const uint4* __restrict__ idx, uint32_t n,
                                               PrimBox* __restrict__ box, uint32_t* __restrict__ prims,
                                               uint32_t* counters, uint32_t* cbk, float rel_pad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t kmn[3] = {fkey(1e34f), fkey(1e34f), fkey(1e34f)}, kmx[3] = {fkey(-1e34f), fkey(-1e34f), fkey(-1e34f)};
  uint32_t cmn[3] = {kmn[0], kmn[1], kmn[2]}, cmx[3] = {kmx[0], kmx[1], kmx[2]};
  if (i < n) {
    const float floor_mag = __fmul_rn(0.25f, __uint_as_float(counters[kMag]));
    const uint4 t = idx[i];
    const float4 a = v[t.x], b = v[t.y], c = v[t.z];
    float mn[3], mx[3], ce[3];
    bool ok = true;
    for (int k = 0; k < 3; k++) {
      const float pa = comp(a, k), pb = comp(b, k), pc = comp(c, k);
      float lo_k = gmin(pa, gmin(pb, pc)), hi_k = gmax(pa, gmax(pb, pc));
      const float pad = __fmul_rn(rel_pad, gmax(floor_mag, gmax(fabsf(lo_k), fabsf(hi_k))));
      lo_k = __fadd_rn(__fsub_rn(lo_k, pad), 0.0f);  // -0 becomes +0
      hi_k = __fadd_rn(__fadd_rn(hi_k, pad), 0.0f);
      mn[k] = lo_k, mx[k] = hi_k;
      ce[k] = __fmul_rn(0.5f, __fadd_rn(lo_k, hi_k));
      ok &= isfinite(lo_k) && isfinite(hi_k) && isfinite(ce[k]);
    }
    if (!ok) atomicOr(&counters[kError], kErrRange);
    box[i] = PrimBox{make_float4(mn[0], mn[1], mn[2], 0.0f), make_float4(mx[0], mx[1], mx[2], 0.0f)};
    prims[i] = i;
    for (int k = 0; k < 3; k++) {
      kmn[k] = fkey(mn[k]), kmx[k] = fkey(mx[k]);
      cmn[k] = min(cmn[k], fkey(ce[k])), cmx[k] = max(cmx[k], fkey(ce[k]));
    }
  }
  block_root_keys(counters + kRootKeys, kmn, kmx);
  __syncthreads();  // its shared words are used again
  block_root_keys(cbk, cmn, cmx);
}

__global__ void k_froot(FNodeD* arena, int32_t* large, int32_t* mid, int32_t* small, uint32_t n, uint32_t mid_most,
                        uint32_t* counters) {
  float mn[3], mx[3];
  for (int k = 0; k < 3; k++) mn[k] = unkey(counters[kRootKeys + k]), mx[k] = unkey(counters[kRootKeys + 3 + k]);
  arena[0] = make_node(mn, mx, 0, n, -1, 0);
  counters[kArenaCount] = 1;
  if (n >= 2) {
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
// they are large and to the final array otherwise, so nothing is copied back, and
// takes the children's centroid bounds on the way. With a copy pass, a pass for the
// bounds and one for the offsets a level of 2.0 M triangles took 128 us, now 94.
struct LevelArgs {
  FNodeD* arena;
  int32_t* large[2];
  uint32_t max_large;
  int32_t* mid;
  uint32_t max_mid, mid_most;
  int32_t* small;
  uint32_t max_small;
  uint32_t* counters;
  uint32_t cap;
  float ascale;
  uint32_t chunk, max_chunks;
  Chunk* chunks;
  FSplit* split;
  uint32_t* bins;
  uint32_t* cbk[2];
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

// One warp per node: its lanes write the chunks and the empty bins (one thread
// took up to 31 us a level over the 336 bin words of its node).
__global__ void __launch_bounds__(256) k_fchunks(LevelArgs A, int par) {
  after_previous();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  // the next level's counters: its last reader was the level before this one
  if (blockIdx.x == 0 && threadIdx.x == 0) A.counters[kLarge + (par ^ 1)] = 0, A.counters[kChunks + (par ^ 1)] = 0;
  if (s >= large_count(A, par)) return;  // whole warp
  const FNodeD& nd = A.arena[A.large[par][s]];
  const uint32_t cnt = (uint32_t)nd.count, nc = (cnt + A.chunk - 1) / A.chunk;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&A.counters[kChunks + par], nc);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (base + nc > A.max_chunks) {
    if (lane == 0) {
      atomicOr(&A.counters[kError], kErrArena);
      A.split[s] = FSplit{-2, {-1, -1}, 0, 0.0f, 0.0f, 0, 0u, 0u};
    }
    for (uint32_t c = base + lane; c < A.max_chunks; c += 32) A.chunks[c] = Chunk{(int32_t)s, 0u, 0u};
    return;
  }
  for (uint32_t c = lane; c < nc; c += 32) {
    const uint32_t b = (uint32_t)nd.first + c * A.chunk;
    A.chunks[base + c] = Chunk{(int32_t)s, b, (uint32_t)nd.first + min(cnt, (c + 1) * A.chunk)};
  }
  if (lane == 0) A.split[s] = FSplit{-1, {-1, -1}, 0, 0.0f, 0.0f, 0, 0u, base};
  uint32_t* b = A.bins + (size_t)s * kBinWords;
  for (int w = lane; w < kBinWords; w += 32) b[w] = bin_init(w);
}

__global__ void __launch_bounds__(256) k_fbin(LevelArgs A, int par) {
  after_previous();
  __shared__ uint32_t bins[kBinWords];
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const uint32_t* prims = A.buf[par];
  float blo[3], bscale[3];
  bin_frame(A.cbk[par] + 6 * (size_t)ch.slot, blo, bscale);
  for (int w = threadIdx.x; w < kBinWords; w += blockDim.x) bins[w] = bin_init(w);
  __syncthreads();
  for (uint32_t k0 = ch.begin; k0 < ch.end; k0 += blockDim.x) {
    const bool in = k0 + threadIdx.x < ch.end;
    const PrimBox v = prim_box(A.box + (in ? prims[k0 + threadIdx.x] : 0u));
    int bin[3];
    bins_of(blo, bscale, centre(v), bin);
    bin_warp(bins, bin, v.lo, v.hi, in);
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

// Allocate the two children of node ni and queue them; their slots go to sp.kid.
__device__ __forceinline__ void add_children(const LevelArgs& A, int par, int32_t ni, const FNodeD& nd, uint32_t mid,
                                             const float lmn[3], const float lmx[3], const float rmn[3],
                                             const float rmx[3], FSplit& sp) {
  const uint32_t cid = atomicAdd(&A.counters[kArenaCount], 2u);
  if (cid + 2 > A.cap) {
    atomicOr(&A.counters[kError], kErrArena);
    return;
  }
  const uint32_t count = (uint32_t)nd.count;
  A.arena[cid] = make_node(lmn, lmx, (uint32_t)nd.first, mid, ni, nd.depth + 1);
  A.arena[cid + 1] = make_node(rmn, rmx, (uint32_t)nd.first + mid, count - mid, ni, nd.depth + 1);
  A.arena[ni].left = (int32_t)cid;
  const int nx = par ^ 1;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const uint32_t c = i ? count - mid : mid;
    if (c <= A.mid_most || nd.depth + 1 >= kDepthLimit) {
      queue_child((int32_t)cid + i, c, nd.depth + 1, A.mid, A.max_mid, A.small, A.max_small, A.counters);
      continue;
    }
    const uint32_t s = atomicAdd(&A.counters[kLarge + nx], 1u);
    if (s >= A.max_large) {
      atomicOr(&A.counters[kError], kErrArena);
      continue;
    }
    A.large[nx][s] = (int32_t)cid + i;
    for (int k = 0; k < 6; k++) A.cbk[nx][6 * (size_t)s + k] = k < 3 ? fkey(1e34f) : fkey(-1e34f);
    sp.kid[i] = (int32_t)s;
  }
}

__global__ void __launch_bounds__(256) k_fsplit(LevelArgs A, int par) {
  after_previous();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (s >= large_count(A, par)) return;  // whole warp
  if (A.split[s].mode == -2) return;     // no chunks (the build fails)
  const int32_t ni = A.large[par][s];
  const FNodeD nd = A.arena[ni];
  float blo[3], bscale[3];
  bin_frame(A.cbk[par] + 6 * (size_t)s, blo, bscale);
  // the candidates walk the bins word by word: from shared memory
  __shared__ uint32_t sbins[8][kBinWords];
  uint32_t* bins = sbins[threadIdx.x >> 5];
  for (int w = lane; w < kBinWords; w += 32) bins[w] = A.bins[(size_t)s * kBinWords + w];
  __syncwarp();
  Cand c;
  choose_bin_split(bins, bscale, A.ascale, lane, c);
  const uint32_t count = (uint32_t)nd.count;
  if (c.j < kCands) {
    if (lane == 0) {
      const int a = c.j / (kBins - 1);
      FSplit sp{0, {-1, -1}, a, blo[a], bscale[a], c.j % (kBins - 1) + 1, c.lc, A.split[s].chunk0};
      add_children(A, par, ni, nd, c.lc, c.lmn, c.lmx, c.rmn, c.rmx, sp);
      A.split[s] = sp;
    }
    return;
  }
  // every centroid in one bin on every axis: halve the range as it lies
  const uint32_t mid = count / 2;
  float lmn[3], lmx[3], rmn[3], rmx[3];
  const uint32_t* prims = A.buf[par];
  warp_union(A.box, prims, (uint32_t)nd.first, (uint32_t)nd.first + mid, lane, lmn, lmx);
  warp_union(A.box, prims, (uint32_t)nd.first + mid, (uint32_t)nd.first + count, lane, rmn, rmx);
  if (lane == 0) {
    FSplit sp{1, {-1, -1}, 0, 0.0f, 0.0f, 0, mid, A.split[s].chunk0};
    add_children(A, par, ni, nd, mid, lmn, lmx, rmn, rmx, sp);
    A.split[s] = sp;
  }
}

// Which side each primitive of a chunk goes to (a bit each), how many go left, and
// the centroid bounds of the children that are split on the next level.
__global__ void __launch_bounds__(256) k_fpcount(LevelArgs A, int par) {
  after_previous();
  __shared__ uint32_t red[2][6], nleft;
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const FSplit sp = A.split[ch.slot];
  if (sp.mode < 0) return;
  const uint32_t* prims = A.buf[par];
  const uint32_t half = (uint32_t)A.arena[A.large[par][ch.slot]].first + sp.lc;  // mode 1: the left half's end
  if (threadIdx.x < 12) red[threadIdx.x / 6][threadIdx.x % 6] = threadIdx.x % 6 < 3 ? 0xffffffffu : 0u;
  if (threadIdx.x == 0) nleft = 0;
  __syncthreads();
  uint32_t key[2][6];
  for (int i = 0; i < 2; i++)
    for (int k = 0; k < 6; k++) key[i][k] = k < 3 ? 0xffffffffu : 0u;
  const int lane = threadIdx.x & 31;
  uint32_t n = 0;
  uint32_t* bits = A.left + (size_t)blockIdx.x * (A.chunk / 32);
  for (uint32_t k0 = ch.begin; k0 < ch.end; k0 += blockDim.x) {
    const uint32_t k = k0 + threadIdx.x;
    const bool in = k < ch.end;
    const float4 c = centre(prim_box(A.box + (in ? prims[k] : 0u)));
    const bool left = in && (sp.mode == 1 ? k < half : bin_of(comp(c, sp.axis), sp.lo, sp.scale) < sp.bsp);
    const bool right = in && !left;
    const uint32_t b = __ballot_sync(0xffffffffu, left);
    if (lane == 0) bits[(k0 - ch.begin + threadIdx.x) / 32] = b, n += __popc(b);
    const uint32_t v[3] = {fkey(c.x), fkey(c.y), fkey(c.z)};
#pragma unroll
    for (int a = 0; a < 3; a++) {
      key[0][a] = min(key[0][a], left ? v[a] : 0xffffffffu), key[0][3 + a] = max(key[0][3 + a], left ? v[a] : 0u);
      key[1][a] = min(key[1][a], right ? v[a] : 0xffffffffu), key[1][3 + a] = max(key[1][3 + a], right ? v[a] : 0u);
    }
  }
  if (lane == 0 && n) atomicAdd(&nleft, n);
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (sp.kid[i] < 0) continue;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const uint32_t mn = __reduce_min_sync(0xffffffffu, key[i][a]), mx = __reduce_max_sync(0xffffffffu, key[i][3 + a]);
      if (lane == 0) atomicMin(&red[i][a], mn), atomicMax(&red[i][3 + a], mx);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) A.chunk_left[blockIdx.x] = nleft;
  if (threadIdx.x < 12) {
    const int i = threadIdx.x / 6, k = threadIdx.x % 6;
    const int32_t kid = i ? sp.kid[1] : sp.kid[0];
    if (kid >= 0) {
      uint32_t* g = A.cbk[par ^ 1] + 6 * (size_t)kid + k;
      if (k < 3) atomicMin(g, red[i][k]);
      else atomicMax(g, red[i][k]);
    }
  }
}

// Stable partition by k_fpcount's bits; every block adds up the node's chunk counts
// before its own. Should they not give the split's left count (they come from the
// same bins), the range stays as it lies and the build fails.
constexpr int kMaxWords = 2048 / 32;  // bit words of a chunk
__global__ void __launch_bounds__(256) k_fpscatter(LevelArgs A, int par) {
  after_previous();
  __shared__ uint32_t word[kMaxWords], before[kMaxWords], sum[2];
  if (blockIdx.x >= chunk_count(A, par)) return;
  const Chunk ch = A.chunks[blockIdx.x];
  const FSplit sp = A.split[ch.slot];
  if (sp.mode < 0) return;
  const FNodeD& nd = A.arena[A.large[par][ch.slot]];
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
  const uint32_t* from = A.buf[par];
  uint32_t* to_l = sp.kid[0] >= 0 ? A.buf[par ^ 1] : A.prims;
  uint32_t* to_r = sp.kid[1] >= 0 ? A.buf[par ^ 1] : A.prims;
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
// slots in their present order, in two arrays that a partition goes between. Children
// of at most kWarpMax go to the final array and the warps' list. The level kernels
// would take five launches a level for them: 20,480 triangles 778 -> 700 us, 2.0 M
// 3.66 -> 3.57 ms. What is left is the bins' instructions (runs of eight primitives
// kept in registers were slower, 538 against 453 us for this kernel of a 2.0 M build).
struct MidNode {
  int32_t node, depth;
  uint32_t first, count;  // first: within the block's range
  uint32_t par;           // which array its slots lie in
  uint32_t cb[6];         // centroid bounds
};
constexpr size_t kMidBytes = (6 * sizeof(float) + sizeof(uint32_t) + 2 * sizeof(uint16_t));  // per primitive

template <uint32_t kMidMax, int kMidThreads>
__global__ void __launch_bounds__(kMidThreads) k_fmid(LevelArgs A) {
  after_previous();
  constexpr uint32_t kMidWords = kMidMax / 32;
  constexpr int kMidStack = kMidMax / (kWarpMax + 1) + 1;  // pending nodes are disjoint
  extern __shared__ float sh[];
  float* bx = sh;  // bx[c * kMidMax + slot]: min x/y/z, max x/y/z
  uint32_t* id = reinterpret_cast<uint32_t*>(bx + 6 * kMidMax);
  uint16_t* ord = reinterpret_cast<uint16_t*>(id + kMidMax);  // two arrays
  __shared__ uint32_t bins[kBinWords];
  __shared__ MidNode stack[kMidStack];
  __shared__ FSplit split;
  __shared__ uint32_t cb[2][6], wleft[kMidWords], before[kMidWords], total;
  __shared__ int s_sp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  auto box_of = [&](uint32_t j) {
    PrimBox v;
    v.lo = make_float4(bx[j], bx[kMidMax + j], bx[2 * kMidMax + j], 0.0f);
    v.hi = make_float4(bx[3 * kMidMax + j], bx[4 * kMidMax + j], bx[5 * kMidMax + j], 0.0f);
    return v;
  };
  // the bounds of a child from its threads' keys
  auto reduce_keys = [&](uint32_t key[6], uint32_t* to) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const uint32_t mn = __reduce_min_sync(0xffffffffu, key[a]), mx = __reduce_max_sync(0xffffffffu, key[3 + a]);
      if (lane == 0) atomicMin(&to[a], mn), atomicMax(&to[3 + a], mx);
    }
  };
  const uint32_t nmid = min(A.counters[kMid], A.max_mid);
  for (uint32_t m = blockIdx.x; m < nmid; m += gridDim.x) {
    const int32_t root = A.mid[m];
    const uint32_t base = (uint32_t)A.arena[root].first, n = (uint32_t)A.arena[root].count;
    if (threadIdx.x < 6) stack[0].cb[threadIdx.x] = threadIdx.x < 3 ? fkey(1e34f) : fkey(-1e34f);
    if (threadIdx.x == 0) {
      stack[0].node = root, stack[0].depth = A.arena[root].depth;
      stack[0].first = 0, stack[0].count = n, stack[0].par = 0;
    }
    for (int w = threadIdx.x; w < kBinWords; w += kMidThreads) bins[w] = bin_init(w);
    __syncthreads();
    {
      uint32_t key[6];
      for (int k = 0; k < 6; k++) key[k] = k < 3 ? 0xffffffffu : 0u;
      for (uint32_t j = threadIdx.x; j < n; j += kMidThreads) {
        const uint32_t p = A.prims[base + j];
        const PrimBox v = prim_box(A.box + p);
        id[j] = p, ord[j] = (uint16_t)j;
        bx[j] = v.lo.x, bx[kMidMax + j] = v.lo.y, bx[2 * kMidMax + j] = v.lo.z;
        bx[3 * kMidMax + j] = v.hi.x, bx[4 * kMidMax + j] = v.hi.y, bx[5 * kMidMax + j] = v.hi.z;
        const float4 c = centre(v);
        const uint32_t x[3] = {fkey(c.x), fkey(c.y), fkey(c.z)};
        for (int a = 0; a < 3; a++) key[a] = min(key[a], x[a]), key[3 + a] = max(key[3 + a], x[a]);
      }
      reduce_keys(key, stack[0].cb);
    }
    __syncthreads();
    int sp = 1;
    while (sp > 0) {
      const MidNode nd = stack[--sp];
      const uint32_t first = nd.first, count = nd.count;
      const uint16_t* from = ord + nd.par * kMidMax;
      float blo[3], bscale[3];
      bin_frame(nd.cb, blo, bscale);
      for (uint32_t k0 = 0; k0 < count; k0 += kMidThreads) {
        const uint32_t k = k0 + threadIdx.x;
        const bool in = k < count;
        if (k0 + 32 * warp >= count) break;  // whole warp
        const PrimBox v = box_of(in ? from[first + k] : 0u);
        int bin[3];
        bins_of(blo, bscale, centre(v), bin);
        bin_warp(bins, bin, v.lo, v.hi, in);
      }
      if (threadIdx.x < 12) cb[threadIdx.x / 6][threadIdx.x % 6] = threadIdx.x % 6 < 3 ? fkey(1e34f) : fkey(-1e34f);
      __syncthreads();
      if (warp == 0) {
        Cand c;
        choose_bin_split(bins, bscale, A.ascale, lane, c);
        int mode = 0;
        if (c.j >= kCands) {  // every centroid in one bin on every axis: halve the range as it lies
          mode = 1;
          c.j = 0, c.lc = count / 2;
          for (int side = 0; side < 2; side++) {
            uint32_t key[6];
            for (int k = 0; k < 6; k++) key[k] = k < 3 ? fkey(1e34f) : fkey(-1e34f);
            for (uint32_t k = (side ? c.lc : 0u) + lane; k < (side ? count : c.lc); k += 32) {
              const PrimBox v = box_of(from[first + k]);
              const uint32_t x[6] = {fkey(v.lo.x), fkey(v.lo.y), fkey(v.lo.z), fkey(v.hi.x), fkey(v.hi.y), fkey(v.hi.z)};
              for (int a = 0; a < 3; a++) key[a] = min(key[a], x[a]), key[3 + a] = max(key[3 + a], x[3 + a]);
            }
            for (int a = 0; a < 3; a++) {
              const float mn = unkey(__reduce_min_sync(0xffffffffu, key[a])),
                          mx = unkey(__reduce_max_sync(0xffffffffu, key[3 + a]));
              if (side) c.rmn[a] = mn, c.rmx[a] = mx;
              else c.lmn[a] = mn, c.lmx[a] = mx;
            }
          }
        }
        if (lane == 0) {
          const int a = c.j / (kBins - 1);
          split = FSplit{mode, {-1, -1}, a, blo[a], bscale[a], c.j % (kBins - 1) + 1, c.lc, 0u};
          // the children: split further here, by a warp, or leaves
          int top = sp;
          const uint32_t cid = atomicAdd(&A.counters[kArenaCount], 2u);
          if (cid + 2 > A.cap) {
            atomicOr(&A.counters[kError], kErrArena);
            split.mode = -1;
          } else {
            const uint32_t g = base + first;
            A.arena[cid] = make_node(c.lmn, c.lmx, g, c.lc, nd.node, nd.depth + 1);
            A.arena[cid + 1] = make_node(c.rmn, c.rmx, g + c.lc, count - c.lc, nd.node, nd.depth + 1);
            A.arena[nd.node].left = (int32_t)cid;
            for (int i = 0; i < 2; i++) {
              const uint32_t cc = i ? count - c.lc : c.lc;
              if (cc > kWarpMax && nd.depth + 1 < kDepthLimit) {
                split.kid[i] = top;  // at most kMidStack pending: ranges of more than kWarpMax, disjoint
                MidNode& q = stack[top++];
                q.node = (int32_t)cid + i, q.depth = nd.depth + 1;
                q.first = first + (i ? c.lc : 0u), q.count = cc, q.par = nd.par ^ 1u;
              } else {
                queue_child((int32_t)cid + i, cc, nd.depth + 1, A.mid, A.max_mid, A.small, A.max_small, A.counters);
              }
            }
          }
          s_sp = top;
        }
      }
      __syncthreads();
      sp = s_sp;
      for (int w = threadIdx.x; w < kBinWords; w += kMidThreads) bins[w] = bin_init(w);
      const FSplit s = split;
      if (s.mode < 0) {  // the build fails
        __syncthreads();
        continue;
      }
      // the stable partition: a bit per primitive, kept in the lane that read it
      uint32_t slot[kMidMax / kMidThreads], bal[kMidMax / kMidThreads], key[2][6];
      for (int i = 0; i < 2; i++)
        for (int k = 0; k < 6; k++) key[i][k] = k < 3 ? 0xffffffffu : 0u;
#pragma unroll
      for (int i = 0; i < (int)(kMidMax / kMidThreads); i++) {
        const uint32_t w = warp + (kMidThreads / 32) * i, k = 32 * w + lane;
        if (32 * w >= count) break;  // whole warp
        const bool in = k < count;
        slot[i] = in ? from[first + k] : 0u;
        const float4 c = centre(box_of(slot[i]));
        const bool left = in && (s.mode == 1 ? k < s.lc : bin_of(comp(c, s.axis), s.lo, s.scale) < s.bsp);
        bal[i] = __ballot_sync(0xffffffffu, left);
        if (lane == 0) wleft[w] = __popc(bal[i]);
        const uint32_t x[3] = {fkey(c.x), fkey(c.y), fkey(c.z)};
        const bool right = in && !left;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          key[0][a] = min(key[0][a], left ? x[a] : 0xffffffffu), key[0][3 + a] = max(key[0][3 + a], left ? x[a] : 0u);
          key[1][a] = min(key[1][a], right ? x[a] : 0xffffffffu), key[1][3 + a] = max(key[1][3 + a], right ? x[a] : 0u);
        }
      }
      if (32u * warp < count) {
        if (s.kid[0] >= 0) reduce_keys(key[0], cb[0]);
        if (s.kid[1] >= 0) reduce_keys(key[1], cb[1]);
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
      if (threadIdx.x >= 32 && threadIdx.x < 44) {
        const int i = (threadIdx.x - 32) / 6, k = (threadIdx.x - 32) % 6;
        const int32_t kid = i ? s.kid[1] : s.kid[0];
        if (kid >= 0) stack[kid].cb[k] = cb[i][k];
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
__device__ __forceinline__ bool goes_left(const PrimBox* box, uint32_t p, const FSplit& sp) {
  return bin_of(comp(centre(prim_box(box + p)), sp.axis), sp.lo, sp.scale) < sp.bsp;
}

// Exact SAH sweep of a range of 2..16 primitives (sweep_split): every split of
// the centroid order (ties by primitive id) on each axis; reorders the range to
// the winning axis' order. Returns the left count and the child boxes.
__device__ __forceinline__ uint32_t sweep_split(const PrimBox* box, uint32_t* prims,
                                                uint32_t first, uint32_t count, float s, int lane,
                                                uint32_t (*ord)[kSweepMax], float lmn[3], float lmx[3],
                                                float rmn[3], float rmx[3]) {
  const bool in = (uint32_t)lane < count;
  const uint32_t p = in ? prims[first + lane] : 0u;
  const float4 pc = in ? centre(prim_box(box + p)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float best = 3e38f;
  int bax = 0;
  uint32_t bmid = count / 2;
  for (int a = 0; a < 3; a++) {
    const float c = comp(pc, a);
    uint32_t r = 0;
    for (uint32_t j = 0; j < count; j++) {
      const float cj = __shfl_sync(0xffffffffu, c, j);
      const uint32_t pj = __shfl_sync(0xffffffffu, p, j);
      r += (cj < c || (cj == c && pj < p)) ? 1u : 0u;
    }
    if (in) ord[a][r] = p;
    __syncwarp();
    // lane r holds the box of the r-th primitive in this axis' order
    float bmn[3] = {1e34f, 1e34f, 1e34f}, bmx[3] = {-1e34f, -1e34f, -1e34f};
    if (in) {
      const PrimBox v = prim_box(box + ord[a][lane]);
      const float4 l = v.lo, h = v.hi;
      bmn[0] = l.x, bmn[1] = l.y, bmn[2] = l.z, bmx[0] = h.x, bmx[1] = h.y, bmx[2] = h.z;
    }
    float pmn[3], pmx[3], smn[3], smx[3];  // inclusive prefix / suffix unions
    for (int k = 0; k < 3; k++) pmn[k] = smn[k] = bmn[k], pmx[k] = smx[k] = bmx[k];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      for (int k = 0; k < 3; k++) {
        const float umn = __shfl_up_sync(0xffffffffu, pmn[k], off), umx = __shfl_up_sync(0xffffffffu, pmx[k], off);
        const float dmn = __shfl_down_sync(0xffffffffu, smn[k], off), dmx = __shfl_down_sync(0xffffffffu, smx[k], off);
        if (lane >= off) pmn[k] = gmin(pmn[k], umn), pmx[k] = gmax(pmx[k], umx);
        if (lane + off < 32) smn[k] = gmin(smn[k], dmn), smx[k] = gmax(smx[k], dmx);
      }
    }
    float lmn_i[3], lmx_i[3];  // union of the first `lane` primitives
    for (int k = 0; k < 3; k++) {
      lmn_i[k] = __shfl_up_sync(0xffffffffu, pmn[k], 1);
      lmx_i[k] = __shfl_up_sync(0xffffffffu, pmx[k], 1);
    }
    const bool cand = lane >= 1 && (uint32_t)lane < count;
    float cost = 0.0f;
    if (cand)
      cost = __fadd_rn(__fmul_rn(farea(lmn_i, lmx_i, s), __uint2float_rn((uint32_t)lane)),
                       __fmul_rn(farea(smn, smx, s), __uint2float_rn(count - (uint32_t)lane)));
    // first lowest cost below the running best, in split order
    float bc = cost;
    int bi = (cand && cost < best) ? lane : 64;
#pragma unroll
    for (int off = 16; off; off >>= 1) {
      const float oc = __shfl_xor_sync(0xffffffffu, bc, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      if (oi < 64 && (bi >= 64 || oc < bc || (oc == bc && oi < bi))) bc = oc, bi = oi;
    }
    if (bi < 64) best = bc, bax = a, bmid = (uint32_t)bi;
  }
  __syncwarp();
  if (in) prims[first + lane] = ord[bax][lane];
  __syncwarp();
  // cut_boxes over the reordered range
  warp_union(box, prims, first, first + bmid, lane, lmn, lmx);
  warp_union(box, prims, first + bmid, first + count, lane, rmn, rmx);
  return bmid;
}

// A subtree of 2..16 primitives goes to k_fleaf when no split of it can reach
// the depth limit (its deepest node of two primitives is at depth + count - 2),
// so that it ends in single primitives and its node count is known.
__device__ __forceinline__ bool leaf_task(uint32_t count, int32_t depth) {
  return count >= 2 && count <= kSweepMax && depth + (int32_t)count - 2 < kDepthLimit;
}

// tasks: ranges for k_fleaf, counted in counters[kTasks]; at most n / 2 of them
// (disjoint, two primitives or more each).
__global__ void __launch_bounds__(kSmallWarps * 32) k_fsmall(LevelArgs A, uint32_t* tasks) {
  const PrimBox* __restrict__ box = A.box;
  uint32_t* prims = A.prims;
  __shared__ uint32_t sbins[kSmallWarps][kBinWords];
  __shared__ int32_t sstack[kSmallWarps][kSmallStack];
  __shared__ uint32_t stmp[kSmallWarps][2 * kWarpMax];
  __shared__ uint32_t sord[kSmallWarps][3][kSweepMax];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* bins = sbins[warp];
  int32_t* stack = sstack[warp];
  uint32_t* tmp = stmp[warp];
  const uint32_t nsmall = min(A.counters[kSmallCount], A.max_small);
  for (uint32_t sidx = blockIdx.x * kSmallWarps + warp; sidx < nsmall; sidx += gridDim.x * kSmallWarps) {
    const int32_t root = A.small[sidx];
    if (leaf_task((uint32_t)A.arena[root].count, A.arena[root].depth)) {
      if (lane == 0) tasks[atomicAdd(&A.counters[kTasks], 1u)] = (uint32_t)root;
      continue;
    }
    if (lane == 0) stack[0] = root;
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
      const int32_t ni = stack[--sp];
      __syncwarp();
      const FNodeD nd = A.arena[ni];
      const uint32_t first = (uint32_t)nd.first, count = (uint32_t)nd.count;
      float lmn[3], lmx[3], rmn[3], rmx[3];
      uint32_t mid;
      if (count <= kSweepMax) {
        mid = sweep_split(box, prims, first, count, A.ascale, lane, sord[warp], lmn, lmx, rmn, rmx);
      } else {
        // centroid bounds, bins, the 45 bin splits
        uint32_t kmn[3] = {fkey(1e34f), fkey(1e34f), fkey(1e34f)}, kmx[3] = {fkey(-1e34f), fkey(-1e34f), fkey(-1e34f)};
        for (uint32_t k = lane; k < count; k += 32) {
          const float4 c = centre(prim_box(box + prims[first + k]));
          kmn[0] = min(kmn[0], fkey(c.x)), kmn[1] = min(kmn[1], fkey(c.y)), kmn[2] = min(kmn[2], fkey(c.z));
          kmx[0] = max(kmx[0], fkey(c.x)), kmx[1] = max(kmx[1], fkey(c.y)), kmx[2] = max(kmx[2], fkey(c.z));
        }
        uint32_t keys[6];
        for (int a = 0; a < 3; a++) {
          keys[a] = __reduce_min_sync(0xffffffffu, kmn[a]);
          keys[3 + a] = __reduce_max_sync(0xffffffffu, kmx[a]);
        }
        float blo[3], bscale[3];
        bin_frame(keys, blo, bscale);
        for (int w = lane; w < kBinWords; w += 32) bins[w] = bin_init(w);
        __syncwarp();
        for (uint32_t k0 = 0; k0 < count; k0 += 32) {
          const bool in = k0 + lane < count;
          const PrimBox v = prim_box(box + (in ? prims[first + k0 + lane] : 0u));
          int bin[3];
          bins_of(blo, bscale, centre(v), bin);
          bin_warp(bins, bin, v.lo, v.hi, in);
        }
        __syncwarp();
        Cand c;
        choose_bin_split(bins, bscale, A.ascale, lane, c);
        if (c.j < kCands) {
          FSplit sp_;
          sp_.axis = c.j / (kBins - 1);
          sp_.lo = blo[sp_.axis];
          sp_.scale = bscale[sp_.axis];
          sp_.bsp = c.j % (kBins - 1) + 1;
          uint32_t nl = 0, nr = 0;
          for (uint32_t k0 = 0; k0 < count; k0 += 32) {
            const uint32_t k = k0 + lane;
            const bool in = k < count;
            const uint32_t p = in ? prims[first + k] : 0u;
            const bool left = in && goes_left(box, p, sp_);
            const uint32_t bl = __ballot_sync(0xffffffffu, left), br = __ballot_sync(0xffffffffu, in && !left);
            if (left) tmp[nl + __popc(bl & lt)] = p;
            else if (in) tmp[kWarpMax + nr + __popc(br & lt)] = p;
            nl += __popc(bl), nr += __popc(br);
          }
          __syncwarp();
          if (nl != c.lc) {
            if (lane == 0) atomicOr(&A.counters[kError], kErrPartition);
            continue;
          }
          for (uint32_t k = lane; k < count; k += 32) prims[first + k] = k < nl ? tmp[k] : tmp[kWarpMax + k - nl];
          mid = nl;
          for (int k = 0; k < 3; k++) lmn[k] = c.lmn[k], lmx[k] = c.lmx[k], rmn[k] = c.rmn[k], rmx[k] = c.rmx[k];
        } else {
          mid = count / 2;
          warp_union(box, prims, first, first + mid, lane, lmn, lmx);
          warp_union(box, prims, first + mid, first + count, lane, rmn, rmx);
        }
      }
      __syncwarp();
      uint32_t cid = 0;
      if (lane == 0) cid = atomicAdd(&A.counters[kArenaCount], 2u);
      cid = __shfl_sync(0xffffffffu, cid, 0);
      if (cid + 2 > A.cap) {
        if (lane == 0) atomicOr(&A.counters[kError], kErrArena);
        continue;
      }
      if (lane == 0) {
        A.arena[cid] = make_node(lmn, lmx, first, mid, ni, nd.depth + 1);
        A.arena[cid + 1] = make_node(rmn, rmx, first + mid, count - mid, ni, nd.depth + 1);
        A.arena[ni].left = (int32_t)cid;
      }
      const bool more = nd.depth + 1 < kDepthLimit;
      const bool task_r = leaf_task(count - mid, nd.depth + 1), task_l = leaf_task(mid, nd.depth + 1);
      const bool push_r = more && count - mid > 1 && !task_r, push_l = more && mid > 1 && !task_l;
      if (lane == 0 && (task_l || task_r)) {
        uint32_t at = atomicAdd(&A.counters[kTasks], (uint32_t)task_l + (uint32_t)task_r);
        if (task_l) tasks[at++] = cid;
        if (task_r) tasks[at] = cid + 1;
      }
      if (sp + (int)push_r + (int)push_l > kSmallStack) {
        if (lane == 0) atomicOr(&A.counters[kError], kErrStack);
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

// ---------------------------------------------------------------- subtrees of at most 16 primitives, one thread each
// The sweep of sweep_split, by one thread for a whole subtree. The range is
// sorted once per axis (centroid, ties by primitive id); an order is 16 nibbles
// of a 64-bit word, and a split partitions the other two orders stably, so
// every node's orders are its sub-ranges' sorted orders. Nodes are numbered as
// they are made and split in that order: the subtree's 2 (count - 1) nodes come
// from the arena in one piece. Boxes lie in shared memory [value][thread], free
// of bank conflicts whatever primitive each thread reads.
//
// One warp per node (sweep_split, kept for subtrees near the depth limit) spends
// its shuffles, scans and latencies on a range of two as on one of sixteen, and
// nine in ten nodes are in such ranges: k_fsmall took 4.33 ms of a 2.0
// M-triangle build by itself; with the leaves here it takes 0.49 and this kernel
// 0.47 ms.
// Few tasks are spread over all resident warps, a few lanes each: a warp is as slow
// as its lanes' different paths added up (a 20,480-triangle build 1,034 us with 32
// tasks to a warp, 991 spread).
constexpr int kLeafThreads = 64;
constexpr int kLeafWords = 16 * 6 + 16 * 3 + 16 + 16;  // boxes, centroids (then right areas), ids, nodes
constexpr size_t kLeafShared = sizeof(float) * kLeafWords * kLeafThreads;

__device__ __forceinline__ uint32_t nib(unsigned long long o, uint32_t i) { return (uint32_t)(o >> (4 * i)) & 15u; }

__global__ void __launch_bounds__(kLeafThreads) k_fleaf(LevelArgs A, const uint32_t* __restrict__ tasks) {
  const PrimBox* __restrict__ boxes = A.box;
  uint32_t* prims = A.prims;
  extern __shared__ float sh[];
  constexpr int T = kLeafThreads;
  float* box = sh + threadIdx.x;                         // box[(6 j + c) T]: min x/y/z, max x/y/z of primitive j
  float* cen = box + 96 * T;                             // cen[(3 j + a) T], later right areas
  uint32_t* id = reinterpret_cast<uint32_t*>(cen + 48 * T);   // id[j T]
  uint32_t* node = id + 16 * T;                          // two nodes per word: b | count << 4 | depth << 9
  const uint32_t ntask = A.counters[kTasks];
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (T / 32), lanes = min(32u, (ntask + warps - 1) / warps);
  for (uint32_t t0 = (blockIdx.x * (T / 32) + (threadIdx.x >> 5)) * lanes; t0 < ntask; t0 += warps * lanes) {
    const bool in = lane < (int)lanes && t0 + lane < ntask;
    const int32_t root = in ? (int32_t)tasks[t0 + lane] : 0;
    uint32_t first = 0, count = 0;
    int32_t depth0 = 0;
    if (in) {
      const FNodeD nd = A.arena[root];
      first = (uint32_t)nd.first, count = (uint32_t)nd.count, depth0 = nd.depth;
    }
    // the warp's nodes from the arena with one atomic
    const uint32_t need = in ? 2u * (count - 1u) : 0u;
    uint32_t inc = need;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += y;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&A.counters[kArenaCount], inc);
    base = __shfl_sync(0xffffffffu, base, 31) + inc - need;
    if (!in) continue;
    if (base + need > A.cap) {
      atomicOr(&A.counters[kError], kErrArena);
      continue;
    }
    for (uint32_t j = 0; j < count; j++) {
      const uint32_t p = prims[first + j];
      const PrimBox v = prim_box(boxes + p);
      const float4 l = v.lo, h = v.hi, c = centre(v);
      float* b = box + 6 * j * T;
      b[0] = l.x, b[T] = l.y, b[2 * T] = l.z, b[3 * T] = h.x, b[4 * T] = h.y, b[5 * T] = h.z;
      float* e = cen + 3 * j * T;
      e[0] = c.x, e[T] = c.y, e[2 * T] = c.z;
      id[j * T] = p;
    }
    unsigned long long ord[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      unsigned long long o = 0;
      for (uint32_t j = 1; j < count; j++) {  // insertion: o's nibbles 0..j-1 are sorted
        const float c = cen[(3 * j + a) * T];
        const uint32_t p = id[j * T];
        uint32_t k = j;
        while (k > 0) {
          const uint32_t q = nib(o, k - 1);
          const float d = cen[(3 * q + a) * T];
          if (d < c || (d == c && id[q * T] < p)) break;
          k--;
        }
        const unsigned long long low = o & ((1ull << (4 * k)) - 1ull);
        o = low | ((unsigned long long)j << (4 * k)) | ((o - low) << 4);
      }
      ord[a] = o;
    }
    float* ra = cen;  // ra[i T]: area of the range's primitives i.. on the axis at hand
    uint32_t made = 1;
    uint16_t* nodes = reinterpret_cast<uint16_t*>(node);
    auto at = [&](uint32_t k) -> uint16_t& { return nodes[2 * ((k >> 1) * T) + (k & 1u)]; };
    at(0) = (uint16_t)(count << 4);
    for (uint32_t k = 0; k < made; k++) {
      const uint32_t w = at(k), b = w & 15u, n = (w >> 4) & 31u, dep = w >> 9;
      if (n < 2) continue;
      const int32_t ni = k == 0 ? root : (int32_t)(base + k - 1);
      float best = 3e38f;
      int bax = 0;
      uint32_t bmid = n / 2;
      for (int a = 0; a < 3; a++) {
        const unsigned long long o = (a == 0 ? ord[0] : a == 1 ? ord[1] : ord[2]) >> (4 * b);
        float mn[3] = {1e34f, 1e34f, 1e34f}, mx[3] = {-1e34f, -1e34f, -1e34f};
        for (uint32_t i = n - 1; i > 0; i--) {
          const float* q = box + 6 * nib(o, i) * T;
          for (int c = 0; c < 3; c++) mn[c] = fminf(mn[c], q[c * T]), mx[c] = fmaxf(mx[c], q[(3 + c) * T]);
          ra[i * T] = farea(mn, mx, A.ascale);
        }
        for (int c = 0; c < 3; c++) mn[c] = 1e34f, mx[c] = -1e34f;
        for (uint32_t i = 1; i < n; i++) {
          const float* q = box + 6 * nib(o, i - 1) * T;
          for (int c = 0; c < 3; c++) mn[c] = fminf(mn[c], q[c * T]), mx[c] = fmaxf(mx[c], q[(3 + c) * T]);
          const float cost = __fadd_rn(__fmul_rn(farea(mn, mx, A.ascale), __uint2float_rn(i)),
                                       __fmul_rn(ra[i * T], __uint2float_rn(n - i)));
          if (cost < best) best = cost, bax = a, bmid = i;
        }
      }
      // the children's boxes, and the other orders partitioned
      const unsigned long long ow = bax == 0 ? ord[0] : bax == 1 ? ord[1] : ord[2];
      float mn[2][3], mx[2][3];
      uint32_t left = 0;  // primitives of the left child
      for (int c = 0; c < 3; c++) mn[0][c] = mn[1][c] = 1e34f, mx[0][c] = mx[1][c] = -1e34f;
      for (uint32_t i = 0; i < n; i++) {
        const uint32_t j = nib(ow, b + i);
        const float* q = box + 6 * j * T;
        if (i < bmid) {
          left |= 1u << j;
          for (int c = 0; c < 3; c++) mn[0][c] = fminf(mn[0][c], q[c * T]), mx[0][c] = fmaxf(mx[0][c], q[(3 + c) * T]);
        } else {
          for (int c = 0; c < 3; c++) mn[1][c] = fminf(mn[1][c], q[c * T]), mx[1][c] = fmaxf(mx[1][c], q[(3 + c) * T]);
        }
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        if (a == bax) continue;
        unsigned long long o = ord[a];
        uint32_t pl = b, pr = b + bmid;
        const unsigned long long src = o;
        for (uint32_t i = 0; i < n; i++) {
          const uint32_t j = nib(src, b + i);
          const uint32_t to = (left >> j) & 1u ? pl++ : pr++;
          o = (o & ~(15ull << (4 * to))) | ((unsigned long long)j << (4 * to));
        }
        ord[a] = o;
      }
      const uint32_t cid = base + made - 1;
      A.arena[cid] = make_node(mn[0], mx[0], first + b, bmid, ni, depth0 + (int32_t)dep + 1);
      A.arena[cid + 1] = make_node(mn[1], mx[1], first + b + bmid, n - bmid, ni, depth0 + (int32_t)dep + 1);
      A.arena[ni].left = (int32_t)cid;
      at(made) = (uint16_t)(b | (bmid << 4) | ((dep + 1) << 9));
      at(made + 1) = (uint16_t)((b + bmid) | ((n - bmid) << 4) | ((dep + 1) << 9));
      made += 2;
    }
    for (uint32_t i = 0; i < count; i++) prims[first + i] = id[nib(ord[0], i) * T];
  }
}

// ---------------------------------------------------------------- cost table
__device__ __forceinline__ void node_cost(const FNodeD& n, const FCostD* cost, float s, FCostD& e) {
  const float A = farea(n.mn, n.mx, s);
  const uint32_t count = (uint32_t)n.count;
  float leaf = 3e38f;
  if (count <= kLeafMax || n.left < 0) leaf = __fmul_rn(A, __uint2float_rn(2u * ((count + 1u) / 2u)));
  float dist[5] = {3e38f, 3e38f, 3e38f, 3e38f, 3e38f};
  uint32_t dk[5] = {0, 0, 0, 0, 0};
  if (n.left >= 0) {
    float L[4], R[4];
    for (int k = 0; k < 4; k++) L[k] = __ldcg(&cost[n.left].c[k]), R[k] = __ldcg(&cost[n.left + 1].c[k]);
    for (int j = 2; j <= 4; j++)
      for (int k = 1; k < j; k++) {
        const float v = __fadd_rn(L[k - 1], R[j - k - 1]);
        if (v < dist[j]) dist[j] = v, dk[j] = (uint32_t)k;
      }
  }
  const float inner = __fadd_rn(A, dist[4]);
  uint32_t meta = leaf <= inner ? 1u : 0u;
  e.c[0] = inner < leaf ? inner : leaf;
  for (int i = 2; i <= 4; i++) {
    if (dist[i] < e.c[i - 2]) {
      e.c[i - 1] = dist[i];
      meta |= dk[i] << (8 * (i - 1));
    } else {
      e.c[i - 1] = e.c[i - 2];
    }
  }
  e.meta = meta;
}

__device__ __forceinline__ void store_cost(FCostD* dst, const FCostD& e) {
  for (int k = 0; k < 4; k++) __stcg(&dst->c[k], e.c[k]);
  __stcg(&dst->meta, e.meta);
}

__global__ void __launch_bounds__(256) k_fcost(const FNodeD* __restrict__ arena, FCostD* cost, uint32_t* arrive,
                                               const uint32_t* counters, uint32_t cap, float s) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(counters[kArenaCount], cap)) return;
  if (arena[i].left >= 0) return;
  FCostD e;
  node_cost(arena[i], cost, s, e);
  store_cost(&cost[i], e);
  int32_t cur = (int32_t)i;
  while (true) {
    const int32_t p = arena[cur].parent;
    if (p < 0) break;
    __threadfence();
    if (atomicAdd(&arrive[p], 1u) == 0) return;  // the sibling's subtree is not finished yet
    __threadfence();
    const FNodeD np = arena[p];
    node_cost(np, cost, s, e);
    store_cost(&cost[p], e);
    cur = p;
  }
}

// ---------------------------------------------------------------- 8-wide cost table
// Relative costs of the wide tree's traversal per unit of surface area: a wide
// node (one 80-byte fetch and eight slot tests) and one triangle of a leaf slot.
constexpr float kWideNodeCost = 1.0f;
constexpr float kWideTriCost = 1.0f;

__device__ __forceinline__ void wide_cost(const FNodeD& n, const WideCost* cost, float s, WideCost& e) {
  const float A = farea(n.mn, n.mx, s);
  const uint32_t count = (uint32_t)n.count;
  const float inf = 3e38f;
  e.split = 0;
  e.pad[0] = e.pad[1] = 0;
  if (n.left < 0) {
    // a binary leaf takes ceil(count / 3) slots of three triangles
    const uint32_t need = (count + 2u) / 3u;
    const float leaf = __fmul_rn(A, __fmul_rn(kWideTriCost, __uint2float_rn(count)));
    for (int i = 1; i <= 8; i++) e.c[i - 1] = (uint32_t)i >= need ? leaf : inf;
    e.leaf1 = 1;
    return;
  }
  float L[8], R[8];
  for (int k = 0; k < 8; k++) L[k] = __ldcg(&cost[n.left].c[k]), R[k] = __ldcg(&cost[n.left + 1].c[k]);
  float dist[9];
  uint32_t dk[9];
  for (int j = 0; j <= 8; j++) dist[j] = inf, dk[j] = 0;
  for (int j = 2; j <= 8; j++)
    for (int k = 1; k < j; k++) {
      const float v = __fadd_rn(L[k - 1], R[j - k - 1]);
      if (v < dist[j]) dist[j] = v, dk[j] = (uint32_t)k;
    }
  const float leaf = count <= 3u ? __fmul_rn(A, __fmul_rn(kWideTriCost, __uint2float_rn(count))) : inf;
  const float inner = __fadd_rn(__fmul_rn(A, kWideNodeCost), dist[8]);
  e.leaf1 = (count <= 3u && leaf <= inner) ? 1u : 0u;
  e.c[0] = e.leaf1 ? leaf : inner;
  for (int i = 2; i <= 8; i++) {
    if (dist[i] < e.c[i - 2]) {
      e.c[i - 1] = dist[i];
      e.split |= dk[i] << (3 * (i - 2));
    } else {
      e.c[i - 1] = e.c[i - 2];
    }
  }
}

__device__ __forceinline__ void store_wide_cost(WideCost* dst, const WideCost& e) {
  for (int k = 0; k < 8; k++) __stcg(&dst->c[k], e.c[k]);
  __stcg(&dst->split, e.split);
  __stcg(&dst->leaf1, e.leaf1);
}

__global__ void __launch_bounds__(256) k_fcost8(const FNodeD* __restrict__ arena, WideCost* cost, uint32_t* arrive,
                                                const uint32_t* counters, uint32_t cap, float s) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(counters[kArenaCount], cap)) return;
  if (arena[i].left >= 0) return;
  WideCost e;
  wide_cost(arena[i], cost, s, e);
  store_wide_cost(&cost[i], e);
  int32_t cur = (int32_t)i;
  while (true) {
    const int32_t p = arena[cur].parent;
    if (p < 0) break;
    __threadfence();
    if (atomicAdd(&arrive[p], 1u) == 0) return;  // the sibling's subtree is not finished yet
    __threadfence();
    const FNodeD np = arena[p];
    wide_cost(np, cost, s, e);
    store_wide_cost(&cost[p], e);
    cur = p;
  }
}

// ---------------------------------------------------------------- collapse
__device__ __forceinline__ uint32_t split_of(uint32_t meta, int i) { return (meta >> (8 * (i - 1))) & 0xffu; }

// emit (bvh_fast.cpp): the slots of quad node n, depth first, then largest box first
// (stable). Returns their number, -1 when the table is not consistent.
__device__ __forceinline__ int quad_slots(const FNodeD* arena, const FCostD* cost, const FNodeD& n, float s,
                                          int32_t sl[4], bool lf[4]) {
  const int32_t L = n.left, R = L + 1;
  if (L < 0) return -1;  // a quad node is an inner binary node
  float best = 3e38f;
  int bk = 1;
  for (int k = 1; k < 4; k++) {
    const float v = __fadd_rn(cost[L].c[k - 1], cost[R].c[4 - k - 1]);
    if (v < best) best = v, bk = k;
  }
  int ns = 0;
  int32_t stn[8];
  int sti[8];
  int sp = 0;
  stn[sp] = R, sti[sp++] = 4 - bk;
  stn[sp] = L, sti[sp++] = bk;
  while (sp > 0) {
    const int32_t x = stn[--sp];
    int i = sti[sp];
    const uint32_t meta = cost[x].meta;
    while (i > 1 && split_of(meta, i) == 0) i--;
    if (i == 1) {
      if (ns < 4) sl[ns] = x, lf[ns] = (meta & 1u) != 0, ns++;
      continue;
    }
    const int k = (int)split_of(meta, i);
    const int32_t xl = arena[x].left;
    if (sp + 2 > 8 || xl < 0) return -1;
    stn[sp] = xl + 1, sti[sp++] = i - k;
    stn[sp] = xl, sti[sp++] = k;
  }
  float ar[4];
  for (int j = 0; j < ns; j++) ar[j] = farea(arena[sl[j]].mn, arena[sl[j]].mx, s);
  for (int j = 1; j < ns; j++) {
    const float a = ar[j];
    const int32_t x = sl[j];
    const bool f = lf[j];
    int k = j;
    while (k > 0 && ar[k - 1] < a) ar[k] = ar[k - 1], sl[k] = sl[k - 1], lf[k] = lf[k - 1], k--;
    ar[k] = a, sl[k] = x, lf[k] = f;
  }
  return ns;
}

// One level; its nodes follow the previous level's, and their number is read on the
// device, so that several levels can be issued together.
__global__ void __launch_bounds__(256) k_fqlevel(const FNodeD* arena, const FCostD* cost, uint32_t* qlist, QRec* qrec,
                                                 int level, uint32_t qcap, uint32_t* counters, float s) {
  after_previous();
  const uint32_t b = level ? counters[kQuadFirst + level] : 0u;
  const uint32_t e = level ? b + counters[kQuadCount + level] : 1u;
  if (blockIdx.x == 0 && threadIdx.x == 0) counters[kQuadFirst + level + 1] = min(e, qcap);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, n = min(e, qcap) - b;
  if ((i & ~31u) >= n) return;  // whole warp
  int32_t sl[4];
  bool lf[4];
  int ns = 0;
  uint32_t inner = 0;
  if (i < n) {
    ns = quad_slots(arena, cost, arena[qlist[b + i]], s, sl, lf);
    if (ns < 0) atomicOr(&counters[kError], kErrQuad);
    for (int j = 0; j < ns; j++) inner += !lf[j];
  }
  uint32_t at_ = e + warp_alloc(&counters[kQuadCount + level + 1], inner);
  if (i >= n || ns < 0) return;
  QRec r;
  r.leafmask = 0;
  r.nk = 0;
  r.size = 0;
  r.rank = 0;
  r.number = 0;
  r.pad[0] = r.pad[1] = r.pad[2] = 0;
  for (int j = 0; j < 4; j++) {
    r.slot[j] = j < ns ? sl[j] : -1;
    r.kid[j] = -1;
    if (j >= ns) continue;
    if (lf[j]) {
      r.leafmask |= 1u << j;
      const uint32_t cnt = (uint32_t)arena[sl[j]].count;
      if (cnt > __ldcg(&counters[kMaxLeaf])) atomicMax(&counters[kMaxLeaf], cnt);  // few raise it
    } else if (at_ >= qcap) {
      atomicOr(&counters[kError], kErrQuad);
    } else {
      qlist[at_] = (uint32_t)sl[j];
      r.kid[j] = (int32_t)at_++;
      r.nk++;
    }
  }
  qrec[b + i] = r;
}

__global__ void k_fqsize(QRec* qrec, uint32_t b, uint32_t e) {
  after_previous();
  const uint32_t q = b + blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= e) return;
  uint32_t sz = 1;
  for (int j = 0; j < 4; j++)
    if (qrec[q].kid[j] >= 0) sz += qrec[qrec[q].kid[j]].size;
  qrec[q].size = sz;
}

__global__ void k_fqrank(QRec* qrec, uint32_t b, uint32_t e) {
  after_previous();
  const uint32_t q = b + blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= e) return;
  uint32_t r = qrec[q].rank + 1;
  for (int j = 0; j < 4; j++) {
    const int32_t k = qrec[q].kid[j];
    if (k < 0) continue;
    qrec[k].rank = r;
    r += qrec[k].size;
  }
}

__global__ void k_fqscatter(const QRec* __restrict__ qrec, uint32_t nq, uint32_t* scan) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const uint32_t r = qrec[q].rank;
  if (r < nq) scan[r] = qrec[q].nk;
}

// exclusive scan of scan[0, n): per block, then the block totals, then the offsets
__global__ void __launch_bounds__(kScanBlock) k_scan_blocks(uint32_t* scan, uint32_t n, uint32_t* sums) {
  __shared__ uint32_t ws[kScanBlock / 32];
  const uint32_t i = blockIdx.x * kScanBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t v = i < n ? scan[i] : 0u;
  uint32_t x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = ws[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += y;
    }
    ws[lane] = w;
  }
  __syncthreads();
  const uint32_t before = warp ? ws[warp - 1] : 0u;
  if (i < n) scan[i] = before + x - v;
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = before + x;
}

__global__ void __launch_bounds__(32) k_scan_sums(uint32_t* sums, uint32_t nb) {
  const int lane = threadIdx.x;
  uint32_t run = 0;
  for (uint32_t b0 = 0; b0 < nb; b0 += 32) {
    const uint32_t b = b0 + lane;
    const uint32_t v = b < nb ? sums[b] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    if (b < nb) sums[b] = run + x - v;
    run += __shfl_sync(0xffffffffu, x, 31);
  }
}

__global__ void __launch_bounds__(kScanBlock) k_scan_add(uint32_t* scan, uint32_t n, const uint32_t* sums) {
  const uint32_t i = blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) scan[i] += sums[blockIdx.x];
}

__global__ void k_fqnum(QRec* qrec, uint32_t nq, const uint32_t* __restrict__ scan) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const uint32_t r = qrec[q].rank;
  uint32_t next = 1 + (r < nq ? scan[r] : 0u);
  for (int j = 0; j < 4; j++) {
    const int32_t k = qrec[q].kid[j];
    if (k >= 0) qrec[k].number = next++;
  }
}

__device__ __forceinline__ void put_slot(QuadNode& d, int j, const float mn[3], const float mx[3], int32_t child,
                                         int32_t count) {
  d.bminx[j] = mn[0], d.bminy[j] = mn[1], d.bminz[j] = mn[2];
  d.bmaxx[j] = mx[0], d.bmaxy[j] = mx[1], d.bmaxz[j] = mx[2];
  d.childs[j] = child;
  d.counts[j] = count;
}

__global__ void k_fqwrite(const FNodeD* __restrict__ arena, const QRec* __restrict__ qrec, uint32_t nq,
                          QuadNode* quad, uint32_t* counters) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const QRec r = qrec[q];
  const float big[3] = {1e34f, 1e34f, 1e34f}, nbig[3] = {-1e34f, -1e34f, -1e34f};
  QuadNode d;
  for (int j = 0; j < 4; j++) {
    if (r.slot[j] < 0) {
      put_slot(d, j, big, nbig, -1, 0);
      continue;
    }
    const FNodeD& c = arena[r.slot[j]];
    if (r.leafmask & (1u << j)) put_slot(d, j, c.mn, c.mx, c.first, c.count);
    else put_slot(d, j, c.mn, c.mx, r.kid[j] >= 0 ? (int32_t)qrec[r.kid[j]].number : -1, -1);
  }
  if (r.number < nq) quad[r.number] = d;
  else atomicOr(&counters[kError], kErrQuad);
}

// a single primitive: one leaf slot under the root
__global__ void k_fqsingle(const FNodeD* __restrict__ arena, QuadNode* quad, uint32_t* counters) {
  const float big[3] = {1e34f, 1e34f, 1e34f}, nbig[3] = {-1e34f, -1e34f, -1e34f};
  QuadNode d;
  put_slot(d, 0, arena[0].mn, arena[0].mx, 0, arena[0].count);
  for (int j = 1; j < 4; j++) put_slot(d, j, big, nbig, -1, 0);
  quad[0] = d;
  counters[kMaxLeaf] = (uint32_t)arena[0].count;
}

unsigned blocks(uint64_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

#define FB_TRY(call)                  \
  do {                                \
    cudaError_t e_ = (call);          \
    if (e_ != cudaSuccess) return e_; \
  } while (0)

cudaError_t read_counters(uint32_t* host, const uint32_t* dev, cudaStream_t s) {
  FB_TRY(cudaMemcpyAsync(host, dev, 4 * kCounterWords, cudaMemcpyDeviceToHost, s));
  return cudaStreamSynchronize(s);
}

}  // namespace

size_t gpu_fbvh_scratch_bytes(uint32_t n, int wide) { return Layout(n, wide).total; }

void gpu_fbvh_binary(void* scratch, uint32_t n, int wide, const void** arena, const uint32_t** prims,
                     const WideCost** cost) {
  const Layout Lo(n, wide);
  *arena = at<FNodeD>(scratch, Lo.arena);
  *prims = at<uint32_t>(scratch, Lo.prims);
  *cost = wide ? at<WideCost>(scratch, Lo.cost) : nullptr;
}

cudaError_t gpu_fbvh_build(const DevScene& sc, void* scratch, uint32_t* hc, cudaStream_t s, GpuBvhResult& r, int wide) {
  const uint32_t n = sc.tri_count;
  const Layout Lo(n, wide);
  uint32_t* counters = at<uint32_t>(scratch, Lo.counters);
  PrimBox* box = at<PrimBox>(scratch, Lo.box);
  uint32_t* prims = at<uint32_t>(scratch, Lo.prims);
  uint32_t* tmp = at<uint32_t>(scratch, Lo.tmp);
  FNodeD* arena = at<FNodeD>(scratch, Lo.arena);
  FCostD* cost = at<FCostD>(scratch, Lo.cost);
  uint32_t* arrive = at<uint32_t>(scratch, Lo.arrive);
  uint32_t* cbk = at<uint32_t>(scratch, Lo.cbk);
  uint32_t* qlist = at<uint32_t>(scratch, Lo.qlist);
  QRec* qrec = at<QRec>(scratch, Lo.qrec);
  uint32_t* scan = at<uint32_t>(scratch, Lo.scan);
  uint32_t* sums = at<uint32_t>(scratch, Lo.sums);
  r = GpuBvhResult{};

  // the levels' second buffer and partition bits lie where the quad phase works later
  LevelArgs A;
  A.arena = arena;
  A.large[0] = at<int32_t>(scratch, Lo.large0), A.large[1] = at<int32_t>(scratch, Lo.large1);
  A.max_large = Lo.max_large;
  A.mid = at<int32_t>(scratch, Lo.mid);
  A.max_mid = Lo.max_mid, A.mid_most = Lo.mid_most;
  A.small = at<int32_t>(scratch, Lo.small);
  A.max_small = Lo.max_small;
  A.counters = counters;
  A.cap = Lo.cap;
  A.ascale = 0.0f;
  A.chunk = Lo.chunk, A.max_chunks = Lo.max_chunks;
  A.chunks = at<Chunk>(scratch, Lo.chunks);
  A.split = at<FSplit>(scratch, Lo.split);
  A.bins = at<uint32_t>(scratch, Lo.bins);
  A.cbk[0] = cbk, A.cbk[1] = cbk + 6 * (size_t)Lo.max_large;
  A.chunk_left = at<uint32_t>(scratch, Lo.chunk_left);
  A.left = qlist;
  A.box = box;
  A.buf[0] = tmp, A.buf[1] = scan;
  A.prims = prims;

  k_finit<<<1, 32, 0, s>>>(counters, cbk);
  k_fmag<<<blocks(n, 256), 256, 0, s>>>(sc.verts, sc.idx, n, counters);
  k_fprep<<<blocks(n, 256), 256, 0, s>>>(sc.verts, sc.idx, n, box, n > Lo.mid_most ? A.buf[0] : prims, counters, cbk,
                                           wide ? 0.0f : kPad);
  k_froot<<<1, 1, 0, s>>>(arena, A.large[0], A.mid, A.small, n, Lo.mid_most, counters);
  FB_TRY(cudaGetLastError());
  FB_TRY(read_counters(hc, counters, s));
  if (hc[kError]) {
    r.error = hc[kError];
    return cudaSuccess;
  }
  float rmn[3], rmx[3];
  for (int k = 0; k < 3; k++) {
    uint32_t a = hc[kRootKeys + k], b = hc[kRootKeys + 3 + k];
    a = (a & 0x80000000u) ? (a & 0x7fffffffu) : ~a;
    b = (b & 0x80000000u) ? (b & 0x7fffffffu) : ~b;
    std::memcpy(&rmn[k], &a, 4);
    std::memcpy(&rmx[k], &b, 4);
  }
  const float ascale = fast_area_scale(rmn, rmx);
  A.ascale = ascale;
  // Up to four levels are issued before the counters are read back (12 us each time),
  // while all their nodes could be large ones: a level that turns out empty costs
  // five launches.
  uint64_t nl = hc[kLarge];
  int par = 0;
  while (nl > 0) {
    int batch = 1;
    while (batch < 4 && (nl << batch) * Lo.mid_most <= n) batch++;
    for (int i = 0; i < batch; i++, par ^= 1) {
      const uint64_t most = std::min<uint64_t>(nl << i, Lo.max_large);
      const unsigned gn = blocks(most * 32, 256);
      const unsigned gc = (unsigned)std::min<uint64_t>((uint64_t)n / Lo.chunk + most + 1, Lo.max_chunks);
      FB_TRY(launch_after(k_fchunks, gn, 256, 0, s, A, par));
      FB_TRY(launch_after(k_fbin, gc, 256, 0, s, A, par));
      FB_TRY(launch_after(k_fsplit, gn, 256, 0, s, A, par));
      FB_TRY(launch_after(k_fpcount, gc, 256, 0, s, A, par));
      FB_TRY(launch_after(k_fpscatter, gc, 256, 0, s, A, par));
    }
    FB_TRY(cudaGetLastError());
    FB_TRY(read_counters(hc, counters, s));
    if (hc[kError]) {
      r.error = hc[kError];
      return cudaSuccess;
    }
    nl = hc[kLarge + par];
  }
  if (hc[kMid] > 0) {
    const unsigned threads = n > kFewMid ? 256 : 512;
    auto kernel = Lo.mid_most == 1024 ? k_fmid<1024, 256> : n > kFewMid ? k_fmid<2048, 256> : k_fmid<2048, 512>;
    const size_t shared = kMidBytes * Lo.mid_most;
    FB_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared));
    FB_TRY(launch_after(kernel, std::min(hc[kMid], Lo.max_mid), threads, shared, s, A));
  }
  if (n >= 2) {
    // how many subtrees the warps have is known on the device
    const unsigned g = (unsigned)std::min<uint64_t>(blocks((uint64_t)n / 2, kSmallWarps), (uint64_t)sm_count() * 16);
    FB_TRY(cudaMemsetAsync(counters + kTasks, 0, 4, s));
    // the levels' first buffer (4 bytes per primitive) is free now: it takes the tasks
    k_fsmall<<<g, kSmallWarps * 32, 0, s>>>(A, tmp);
    FB_TRY(cudaGetLastError());
    FB_TRY(cudaFuncSetAttribute(k_fleaf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLeafShared));
    int per_sm = 0;
    FB_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fleaf, kLeafThreads, kLeafShared));
    const unsigned gl = (unsigned)std::min<uint64_t>(blocks((uint64_t)n / 2 + 1, kLeafThreads / 32),
                                                     (uint64_t)sm_count() * std::max(1, per_sm));
    k_fleaf<<<gl, kLeafThreads, kLeafShared, s>>>(A, tmp);
    FB_TRY(cudaGetLastError());
  }
  FB_TRY(read_counters(hc, counters, s));
  if (hc[kError]) {
    r.error = hc[kError];
    return cudaSuccess;
  }
  const uint32_t nb = hc[kArenaCount];
  r.binary_nodes = nb;
  if (n == 1) {
    r.quad_nodes = 1;
    r.depth = 1;
    r.max_leaf = 1;
    return cudaSuccess;
  }
  FB_TRY(cudaMemsetAsync(arrive, 0, 4 * (size_t)nb, s));
  if (wide) {
    k_fcost8<<<blocks(nb, 256), 256, 0, s>>>(arena, at<WideCost>(scratch, Lo.cost), arrive, counters, Lo.cap, ascale);
    FB_TRY(cudaGetLastError());
    FB_TRY(read_counters(hc, counters, s));
    r.error = hc[kError];
    return cudaSuccess;
  }
  k_fcost<<<blocks(nb, 256), 256, 0, s>>>(arena, cost, arrive, counters, Lo.cap, ascale);
  // quad levels from the root (binary node 0)
  FB_TRY(cudaMemsetAsync(qlist, 0, 4, s));
  FB_TRY(cudaMemsetAsync(counters + kCounterWords, 0, 4 * (kAllWords - kCounterWords), s));
  std::vector<uint32_t> off{0u, 1u};
  // four levels per readback: their grids are bounds, a level has at most four times
  // the nodes of the one before
  while (off.back() > off[off.size() - 2]) {
    const int l0 = (int)off.size() - 2, batch = std::min(4, kQuadLevels - 1 - l0);
    if (batch <= 0) {
      r.error = kErrQuad;
      return cudaSuccess;
    }
    for (int i = 0; i < batch; i++) {
      const uint64_t most = std::min<uint64_t>((uint64_t)(off[l0 + 1] - off[l0]) << (2 * i), n);
      FB_TRY(launch_after(k_fqlevel, blocks(most, 256), 256, 0, s, arena, cost, qlist, qrec, l0 + i, Lo.qcap, counters,
                          ascale));
    }
    FB_TRY(cudaMemcpyAsync(hc + kCounterWords, counters + kQuadCount + l0 + 1, 4 * (size_t)batch, cudaMemcpyDeviceToHost,
                           s));
    FB_TRY(read_counters(hc, counters, s));
    if (hc[kError]) {
      r.error = hc[kError];
      return cudaSuccess;
    }
    for (int i = 0; i < batch && off.back() > off[off.size() - 2]; i++)
      off.push_back(off.back() + hc[kCounterWords + i]);
  }
  const uint32_t nq = off.back();
  const size_t nlev = off.size() - 2;  // levels with nodes
  for (size_t l = nlev; l-- > 0;)
    FB_TRY(launch_after(k_fqsize, blocks(off[l + 1] - off[l], 256), 256, 0, s, qrec, off[l], off[l + 1]));
  for (size_t l = 0; l < nlev; l++)
    FB_TRY(launch_after(k_fqrank, blocks(off[l + 1] - off[l], 256), 256, 0, s, qrec, off[l], off[l + 1]));
  k_fqscatter<<<blocks(nq, 256), 256, 0, s>>>(qrec, nq, scan);
  const uint32_t nsb = blocks(nq, kScanBlock);
  k_scan_blocks<<<nsb, kScanBlock, 0, s>>>(scan, nq, sums);
  k_scan_sums<<<1, 32, 0, s>>>(sums, nsb);
  k_scan_add<<<nsb, kScanBlock, 0, s>>>(scan, nq, sums);
  k_fqnum<<<blocks(nq, 256), 256, 0, s>>>(qrec, nq, scan);
  FB_TRY(cudaGetLastError());
  FB_TRY(read_counters(hc, counters, s));
  r.error = hc[kError];
  r.quad_nodes = nq;
  r.depth = (uint32_t)nlev;
  r.max_leaf = hc[kMaxLeaf];
  return cudaSuccess;
}

cudaError_t gpu_fbvh_emit(const DevScene& sc, void* scratch, const GpuBvhResult& r, uint32_t leaf_shift,
                          QNodeDev* nodes, float4* tris, uint32_t* prims_out, cudaStream_t s) {
  const uint32_t n = sc.tri_count;
  const Layout Lo(n);
  uint32_t* counters = at<uint32_t>(scratch, Lo.counters);
  const FNodeD* arena = at<FNodeD>(scratch, Lo.arena);
  const QRec* qrec = at<QRec>(scratch, Lo.qrec);
  const uint32_t* prims = at<uint32_t>(scratch, Lo.prims);
  QuadNode* quad = reinterpret_cast<QuadNode*>(nodes);  // until launch_quad_to_dev
  if (n == 1) k_fqsingle<<<1, 1, 0, s>>>(arena, quad, counters);
  else k_fqwrite<<<blocks(r.quad_nodes, 256), 256, 0, s>>>(arena, qrec, r.quad_nodes, quad, counters);
  FB_TRY(cudaGetLastError());
  FB_TRY(launch_quad_to_dev(nodes, r.quad_nodes, leaf_shift, s));
  FB_TRY(launch_leaf_tris(sc, prims, n, tris, s));
  return cudaMemcpyAsync(prims_out, prims, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s);
}

uint32_t gpu_fbvh_error(void* scratch, uint32_t n, uint32_t* hc, cudaStream_t s) {
  const Layout Lo(n);  // quad mode (the wide mode reports its errors from gpu_fbvh_build)
  if (read_counters(hc, at<uint32_t>(scratch, Lo.counters), s) != cudaSuccess) return 0xffffffffu;
  return hc[kError];
}

}  // namespace ct

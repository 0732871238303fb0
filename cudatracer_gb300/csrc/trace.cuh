// Device BVH traversal: closest hit and any hit over the quad tree.
//
// Arithmetic is written with round-to-nearest intrinsics so no multiply-add is
// ever fused, whatever the translation unit's -fmad setting: every slab and
// Moller-Trumbore quantity is computed with the same IEEE single-precision
// operations, in the same order, as the reference's glm code
// (src/BVH/MBVHNode.cuh:69-110, src/Core/Triangle.cuh:13-44), which is what
// makes closest-hit primitive ids and t bit-exact against it.
//
// Min/max: glm::min(x,y) = y < x ? y : x and glm::max(x,y) = x < y ? y : x.
// Hardware min/max agree with them except on NaN (a zero direction component
// with the origin exactly on a bounding plane) and when two zeros of opposite
// sign meet (an origin on two planes). The fast path (FASTMM) uses hardware
// min/max throughout; the exact path uses it where the two agree (inner_step).
// FASTMM traversal also computes each slab plane with one fused multiply-add
// and, for closest hit, visits hit children in true distance order
// (inner_step_sorted) instead of the reference's partial order network: the
// same nearest hit up to exact ties and the rounding of box distances, fewer
// instructions per node.
//
// What bounds it, and the shape that follows. A divergent load takes one pass
// through the L1 data pipe per distinct 128-byte line and lane whatever its
// width, and a missed 32-byte sector about 1.5 passes (measured with random
// lines on GB300), so a ray step reads its 128-byte node, or the next two
// triangles of its leaf, with four 32-byte loads instead of up to eight 16-byte
// ones. Both kinds of step start from the same four loads (Fetch), so a warp
// whose lanes are at nodes and at leaves waits for memory once per round. The
// plane distances of two children are one packed f32x2 instruction, and the
// exact path takes hardware min/max wherever they give the reference's bits
// (inner_step). Against 16-byte loads, separate leaf loads and compare-select
// min/max: closest hit on an 81,920-triangle sphere, 4.2 M rays, 1,553 -> 1,204
// us, 65,536 rays 218 -> 145 us; 641x360 exact frames 303 -> 241 us each;
// 1920x1080 frames on 3.1 M triangles 1.80 -> 1.68 ms each.
#pragma once

#include "ct_internal.h"
#include "vmath.cuh"

namespace ct {

__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// One child's slab interval, reference order: x, then y, then z.
__device__ __forceinline__ void slab(float bminx, float bmaxx, float bminy, float bmaxy, float bminz, float bmaxz,
                                     float ox, float oy, float oz, float ix, float iy, float iz, float& tmin,
                                     float& tmax) {
  float t1 = fmul(fsub(bminx, ox), ix), t2 = fmul(fsub(bmaxx, ox), ix);
  tmin = gmin(t1, t2);
  tmax = gmax(t1, t2);
  t1 = fmul(fsub(bminy, oy), iy);
  t2 = fmul(fsub(bmaxy, oy), iy);
  tmin = gmax(tmin, gmin(t1, t2));
  tmax = gmin(tmax, gmax(t1, t2));
  t1 = fmul(fsub(bminz, oz), iz);
  t2 = fmul(fsub(bmaxz, oz), iz);
  tmin = gmax(tmin, gmin(t1, t2));
  tmax = gmin(tmax, gmax(t1, t2));
}

// Two floats in one 64-bit register pair and the packed operations on them:
// each half is the scalar operation, rounded to nearest.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// 32 bytes of read-only memory in one load; p is 32-byte aligned. Volatile so
// that the loads of a step are issued together, before the branch on its kind.
__device__ __forceinline__ void ldg256(const float4* p, float4& a, float4& b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
               : "l"(p));
}

// 32 bytes as ldg256, by the lanes whose ref is at least `least`.
__device__ __forceinline__ void ldg256_from(int ref, int least, const float4* p, float4& a, float4& b) {
  asm volatile("{ .reg .pred q; setp.ge.s32 q, %9, %10; @q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8]; }"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
               : "l"(p), "r"(ref), "r"(least));
}

// What one ray step reads. Inner node: x planes (min, max of the four children), y
// planes, z planes, child references. Leaf: the next two triangles (kTriFloat4), the
// first's 64 bytes and the upper half of the second's, so 96 bytes of memory for two
// (a leaf with one left reads past it: the array has room for one record beyond its
// last). With both whole records, 128 bytes, trees whose triangles don't stay in L2
// waited for memory: 1 M rays, 4 M-triangle soup on the reference's tree, closest hit
// 7.98 -> 7.07 ms, any hit 6.81 -> 4.42.
// LONE: a leaf with one triangle left reads that one only. A leaf reference is negative
// with its count above the first triangle's index, so one comparison tells. Where trees
// lie in DRAM the second sector costs: 4 M rays, 10 M-triangle soup on the reference's
// tree 43.6 -> 39.2 ms, any hit 35.4 -> 32.4 (with records of 48 bytes 42.8 and 33.9).
// Frames, whose trees stay in L2, lose by the predicate (960x540 4.27 -> 4.34 ms).
struct Fetch {
  float4 v0, v1, v2, v3, v4, v5, v6;
};
template <bool LONE>
__device__ __forceinline__ void fetch(const DevBVH& b, int ref, Fetch& f) {
  const float4* p = ref >= 0 ? reinterpret_cast<const float4*>(b.nodes + ref)
                             : b.tris + kTriFloat4 * (size_t)((uint32_t)ref & b.first_mask);
  float4 unused;
  ldg256(p, f.v0, f.v1);
  ldg256(p + 2, f.v2, f.v3);
  ldg256_from(ref, 0, p + 4, f.v4, f.v5);
  if (LONE) ldg256_from(ref, (int)(0x80000000u + (2u << b.leaf_shift)), p + 6, f.v6, unused);
  else ldg256(p + 6, f.v6, unused);
}

// Moller-Trumbore with the reference's absolute epsilon. Returns the new t
// through `t` when the hit is closer (t' > eps && t > t').
__device__ __forceinline__ bool tri_test(const float4 a, const float4 e1v, const float4 e2v, float ox, float oy,
                                         float oz, float dx, float dy, float dz, float eps, float& t) {
  const float e1x = e1v.x, e1y = e1v.y, e1z = e1v.z;
  const float e2x = e2v.x, e2y = e2v.y, e2z = e2v.z;
  // h = cross(dir, edge2)
  const float hx = fsub(fmul(dy, e2z), fmul(e2y, dz));
  const float hy = fsub(fmul(dz, e2x), fmul(e2z, dx));
  const float hz = fsub(fmul(dx, e2y), fmul(e2x, dy));
  const float det = fadd(fadd(fmul(e1x, hx), fmul(e1y, hy)), fmul(e1z, hz));
  if (det > -eps && det < eps) return false;
  const float f = __frcp_rn(det);
  const float sx = fsub(ox, a.x), sy = fsub(oy, a.y), sz = fsub(oz, a.z);
  const float u = fmul(f, fadd(fadd(fmul(sx, hx), fmul(sy, hy)), fmul(sz, hz)));
  if (u < 0.0f || u > 1.0f) return false;
  // q = cross(s, edge1)
  const float qx = fsub(fmul(sy, e1z), fmul(e1y, sz));
  const float qy = fsub(fmul(sz, e1x), fmul(e1z, sx));
  const float qz = fsub(fmul(sx, e1y), fmul(e1x, sy));
  const float v = fmul(f, fadd(fadd(fmul(dx, qx), fmul(dy, qy)), fmul(dz, qz)));
  if (v < 0.0f || fadd(u, v) > 1.0f) return false;
  const float tt = fmul(f, fadd(fadd(fmul(e2x, qx), fmul(e2y, qy)), fmul(e2z, qz)));
  if (tt > eps && t > tt) {
    t = tt;
    return true;
  }
  return false;
}

// Per-ray traversal state.
struct RayState {
  float ox, oy, oz, dx, dy, dz, ix, iy, iz, t;
  float nox, noy, noz;  // -o * inv, read by the fast-math slab only
  int hit, sp, ref;
  bool odd;  // the exact slab may meet a NaN (inner_step); read by the exact path only
};

// A slab term is NaN only as 0 * inf, inf - inf or from a NaN input: never for a
// finite origin and finite reciprocals on finite planes. (An infinite direction component
// has the reciprocal 0, which a plane distance that overflows could meet; such a ray hits
// no triangle whatever the boxes say.)
__device__ __forceinline__ void ray_begin(const DevBVH& b, RayState& r, float4 o, float4 d, float t0) {
  r.ox = o.x, r.oy = o.y, r.oz = o.z, r.dx = d.x, r.dy = d.y, r.dz = d.z;
  r.ix = __frcp_rn(d.x), r.iy = __frcp_rn(d.y), r.iz = __frcp_rn(d.z);
  r.nox = -o.x * r.ix, r.noy = -o.y * r.iy, r.noz = -o.z * r.iz;
  const float big = 3.4028235e38f;  // the largest float
  r.odd = b.odd || !(fabsf(r.ix) <= big && fabsf(r.iy) <= big && fabsf(r.iz) <= big && fabsf(o.x) <= big &&
                     fabsf(o.y) <= big && fabsf(o.z) <= big);
  r.t = t0;
  r.hit = -1;
  r.sp = 0;
  r.ref = 0;  // root: inner node 0 (the reference's todo[0] = {0, -1})
}

enum StepResult { kContinue = 0, kDone = 1, kOverflow = 2 };

// Plane distances of the four children on one axis. FMA (fast math): one fused
// multiply-add, b * inv + (-o * inv); a zero direction component makes the axis
// NaN, which the hardware min/max drop: the axis then culls nothing (more boxes
// visited, never a hit lost). Otherwise (b - o) * inv as the reference rounds it.
template <bool FMA>
__device__ __forceinline__ void axis_planes(float4& lo, float4& hi, float inv, float off) {
  const f32x2 ii = pack2(inv, inv), oo = pack2(off, off);
  auto t = [&](f32x2 b) { return FMA ? fma2(b, ii, oo) : mul2(add2(b, oo), ii); };
  unpack2(t(pack2(lo.x, lo.y)), lo.x, lo.y);
  unpack2(t(pack2(lo.z, lo.w)), lo.z, lo.w);
  unpack2(t(pack2(hi.x, hi.y)), hi.x, hi.y);
  unpack2(t(pack2(hi.z, hi.w)), hi.z, hi.w);
}
__device__ __forceinline__ void interval(float x1, float x2, float y1, float y2, float z1, float z2, float& tn,
                                         float& tf) {
  tn = max3(fminf(x1, x2), fminf(y1, y2), fminf(z1, z2));
  tf = min3(fmaxf(x1, x2), fmaxf(y1, y2), fmaxf(z1, z2));
}
// The four child intervals of a node with hardware min/max.
template <bool FMA>
__device__ __forceinline__ void slab4(Fetch f, const RayState& r, float& tn0, float& tn1, float& tn2, float& tn3,
                                      float& tf0, float& tf1, float& tf2, float& tf3) {
  axis_planes<FMA>(f.v0, f.v1, r.ix, FMA ? r.nox : -r.ox);
  axis_planes<FMA>(f.v2, f.v3, r.iy, FMA ? r.noy : -r.oy);
  axis_planes<FMA>(f.v4, f.v5, r.iz, FMA ? r.noz : -r.oz);
  interval(f.v0.x, f.v1.x, f.v2.x, f.v3.x, f.v4.x, f.v5.x, tn0, tf0);
  interval(f.v0.y, f.v1.y, f.v2.y, f.v3.y, f.v4.y, f.v5.y, tn1, tf1);
  interval(f.v0.z, f.v1.z, f.v2.z, f.v3.z, f.v4.z, f.v5.z, tn2, tf2);
  interval(f.v0.w, f.v1.w, f.v2.w, f.v3.w, f.v4.w, f.v5.w, tn3, tf3);
}
// The same intervals with the reference's compare-select min/max, the planes
// read again (rare: see inner_step).
__device__ __forceinline__ void slab4_ref(const DevBVH& b, const RayState& r, float& tn0, float& tn1, float& tn2,
                                          float& tn3, float& tf0, float& tf1, float& tf2, float& tf3) {
  const QNodeDev* n = b.nodes + r.ref;
  const float4 x0 = __ldg(&n->bminx), x1 = __ldg(&n->bmaxx);
  const float4 y0 = __ldg(&n->bminy), y1 = __ldg(&n->bmaxy);
  const float4 z0 = __ldg(&n->bminz), z1 = __ldg(&n->bmaxz);
  slab(x0.x, x1.x, y0.x, y1.x, z0.x, z1.x, r.ox, r.oy, r.oz, r.ix, r.iy, r.iz, tn0, tf0);
  slab(x0.y, x1.y, y0.y, y1.y, z0.y, z1.y, r.ox, r.oy, r.oz, r.ix, r.iy, r.iz, tn1, tf1);
  slab(x0.z, x1.z, y0.z, y1.z, z0.z, z1.z, r.ox, r.oy, r.oz, r.ix, r.iy, r.iz, tn2, tf2);
  slab(x0.w, x1.w, y0.w, y1.w, z0.w, z1.w, r.ox, r.oy, r.oz, r.ix, r.iy, r.iz, tn3, tf3);
}

// Compare-and-swap of (distance, child) pairs: the nearer pair goes first.
__device__ __forceinline__ void cas_pair(float& ka, int& ca, float& kb, int& cb) {
  const bool sw = kb < ka;
  const float k = sw ? kb : ka;
  const int c = sw ? cb : ca;
  kb = sw ? ka : kb;
  cb = sw ? ca : cb;
  ka = k;
  ca = c;
}

// Fast-math closest-hit node step: the hit children in true distance order (a
// full 4-sort of (tmin, child) pairs, misses last as +inf), nearest visited
// next and the others pushed far to near with predicated stores. Frames in
// fast math do not reproduce the reference's visiting order, only its nearest
// hit, which no order changes beyond exact ties.
__device__ __forceinline__ StepResult inner_step_sorted(const Fetch& f, RayState& r, int* stack, int stride,
                                                        int limit) {
  float tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3;
  slab4<true>(f, r, tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3);
  int c0 = __float_as_int(f.v6.x), c1 = __float_as_int(f.v6.y), c2 = __float_as_int(f.v6.z),
      c3 = __float_as_int(f.v6.w);
  const float t = r.t, inf = __int_as_float(0x7f800000);
  // a hit child's entry distance is below t, so finite or -inf; misses sort last
  float k0 = (tf0 > 0.0f && tn0 <= tf0 && tn0 < t && c0 != kEmptyChild) ? tn0 : inf;
  float k1 = (tf1 > 0.0f && tn1 <= tf1 && tn1 < t && c1 != kEmptyChild) ? tn1 : inf;
  float k2 = (tf2 > 0.0f && tn2 <= tf2 && tn2 < t && c2 != kEmptyChild) ? tn2 : inf;
  float k3 = (tf3 > 0.0f && tn3 <= tf3 && tn3 < t && c3 != kEmptyChild) ? tn3 : inf;
  cas_pair(k0, c0, k1, c1);
  cas_pair(k2, c2, k3, c3);
  cas_pair(k0, c0, k2, c2);
  cas_pair(k1, c1, k3, c3);
  cas_pair(k1, c1, k2, c2);
  if (!(k0 < inf)) {
    if (r.sp == 0) return kDone;
    r.ref = stack[--r.sp * stride];
    return kContinue;
  }
  if (k1 < inf) {
    if (r.sp + 1 + (int)(k2 < inf) + (int)(k3 < inf) > limit) return kOverflow;
    if (k3 < inf) stack[r.sp++ * stride] = c3;
    if (k2 < inf) stack[r.sp++ * stride] = c2;
    stack[r.sp++ * stride] = c1;
  }
  r.ref = c0;
  return kContinue;
}

// Compare-and-swap of (packed distance, child) pairs as the reference's network
// swaps them: on a > b, so a NaN stays where it is.
__device__ __forceinline__ void cas_packed(float& pa, int& ca, float& pb, int& cb) {
  const bool sw = pa > pb;
  const float p = sw ? pb : pa;
  const int c = sw ? cb : ca;
  pb = sw ? pa : pb;
  cb = sw ? ca : cb;
  pa = p;
  ca = c;
}

// The child id in the low two bits of tmin (MBVHNode.cuh:91-94).
__device__ __forceinline__ float with_id(float tn, int id) { return __int_as_float((__float_as_int(tn) & ~3) | id); }

// Visit the inner node r.ref: slab-test the four children (MBVHNode.cuh:69-110),
// then continue with the nearest hit child and push the others far to near
// (:153-161), in the order the reference's network leaves the four packed tmin
// values in; a missed child's reference is replaced by kEmptyChild and swapped
// along, so what is left at a position says whether it is pushed. The hardware
// min/max equal the reference's compare-select except on NaN (rays marked odd)
// and for the sign of a zero, which shows in a packed tmin of magnitude below 4
// denormal steps only (an origin exactly on a box plane): those nodes take the
// compare-select slabs.
__device__ __forceinline__ StepResult inner_step(const DevBVH& b, const Fetch& f, RayState& r, int* stack, int stride,
                                                 int limit) {
  float tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3;
  slab4<false>(f, r, tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3);
  const float tiny = __int_as_float(4);
  if (r.odd || fminf(min3(fabsf(tn0), fabsf(tn1), fabsf(tn2)), fabsf(tn3)) < tiny)
    slab4_ref(b, r, tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3);
  float p0 = with_id(tn0, 0), p1 = with_id(tn1, 1), p2 = with_id(tn2, 2), p3 = with_id(tn3, 3);
  const float t = r.t;
  // hit test by child slot (MBVHNode.cuh:96); empty slots are never pushed
  int c0 = (tf0 > 0.0f && p0 <= tf0 && p0 < t) ? __float_as_int(f.v6.x) : kEmptyChild;
  int c1 = (tf1 > 0.0f && p1 <= tf1 && p1 < t) ? __float_as_int(f.v6.y) : kEmptyChild;
  int c2 = (tf2 > 0.0f && p2 <= tf2 && p2 < t) ? __float_as_int(f.v6.z) : kEmptyChild;
  int c3 = (tf3 > 0.0f && p3 <= tf3 && p3 < t) ? __float_as_int(f.v6.w) : kEmptyChild;
  // the reference's 5-exchange network, last pair (2,3) (MBVHNode.cuh:98-107)
  cas_packed(p0, c0, p1, c1);
  cas_packed(p2, c2, p3, c3);
  cas_packed(p0, c0, p2, c2);
  cas_packed(p1, c1, p3, c3);
  cas_packed(p2, c2, p3, c3);
  const bool h0 = c0 != kEmptyChild, h1 = c1 != kEmptyChild, h2 = c2 != kEmptyChild, h3 = c3 != kEmptyChild;
  if (!(h0 || h1 || h2 || h3)) {
    if (r.sp == 0) return kDone;
    r.ref = stack[--r.sp * stride];
    return kContinue;
  }
  if (r.sp + (int)h0 + (int)h1 + (int)h2 + (int)h3 - 1 > limit) return kOverflow;
  if (h3 && (h0 || h1 || h2)) stack[r.sp++ * stride] = c3;
  if (h2 && (h0 || h1)) stack[r.sp++ * stride] = c2;
  if (h1 && h0) stack[r.sp++ * stride] = c1;
  r.ref = h0 ? c0 : (h1 ? c1 : (h2 ? c2 : c3));
  return kContinue;
}

// Any-hit variant of inner_step: whether the ray is occluded does not depend
// on the order in which hit children are visited (every node whose packed
// interval passes the reference's test is visited until a triangle hits), so
// the order network is skipped: the lowest hit slot continues, the others are
// pushed.
template <bool FASTMM>
__device__ __forceinline__ StepResult inner_step_any(const DevBVH& b, const Fetch& f, RayState& r, int* stack,
                                                     int stride, int limit) {
  float tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3;
  slab4<FASTMM>(f, r, tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3);
  // the sign of a zero tmin changes no hit test, so only NaN needs the compare-select slabs
  if (!FASTMM && r.odd) slab4_ref(b, r, tn0, tn1, tn2, tn3, tf0, tf1, tf2, tf3);
  const int c0 = __float_as_int(f.v6.x), c1 = __float_as_int(f.v6.y), c2 = __float_as_int(f.v6.z),
            c3 = __float_as_int(f.v6.w);
  const float p0 = with_id(tn0, 0), p1 = with_id(tn1, 1), p2 = with_id(tn2, 2), p3 = with_id(tn3, 3);
  const float t = r.t;
  const bool h0 = tf0 > 0.0f && p0 <= tf0 && p0 < t && c0 != kEmptyChild;
  const bool h1 = tf1 > 0.0f && p1 <= tf1 && p1 < t && c1 != kEmptyChild;
  const bool h2 = tf2 > 0.0f && p2 <= tf2 && p2 < t && c2 != kEmptyChild;
  const bool h3 = tf3 > 0.0f && p3 <= tf3 && p3 < t && c3 != kEmptyChild;
  if (!(h0 || h1 || h2 || h3)) {
    if (r.sp == 0) return kDone;
    r.ref = stack[--r.sp * stride];
    return kContinue;
  }
  // the lowest hit slot continues; the others (never slot 0) are pushed in slot order
  if (r.sp + (int)h0 + (int)h1 + (int)h2 + (int)h3 - 1 > limit) return kOverflow;
  if (h1 && h0) stack[r.sp++ * stride] = c1;
  if (h2 && (h0 || h1)) stack[r.sp++ * stride] = c2;
  if (h3 && (h0 || h1 || h2)) stack[r.sp++ * stride] = c3;
  r.ref = h0 ? c0 : (h1 ? c1 : (h2 ? c2 : c3));
  return kContinue;
}

// Test the leaf r.ref's next two triangles (in primitive order, already
// fetched), then pop; the rest of the leaf stays in r.ref (first + 2, count - 2),
// so a round is not held up by the warp's largest leaf.
template <bool ANY>
__device__ __forceinline__ StepResult leaf_step(const DevBVH& b, const Fetch& f, RayState& r, float eps, int* stack,
                                                int stride) {
  const uint32_t u = (uint32_t)r.ref;
  const uint32_t cnt = (u >> b.leaf_shift) & b.count_mask;
  const float4 a1 = make_float4(f.v1.x, f.v1.y, f.v2.x, 0.0f), a2 = make_float4(f.v2.y, f.v2.z, f.v2.w, 0.0f);
  const float4 b1 = make_float4(f.v1.z, f.v1.w, f.v6.x, 0.0f), b2 = make_float4(f.v6.y, f.v6.z, f.v6.w, 0.0f);
  if (cnt > 0 && tri_test(f.v0, a1, a2, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, eps, r.t)) {
    r.hit = __float_as_int(f.v0.w);
    if (ANY) return kDone;
  }
  if (cnt > 1 && tri_test(f.v3, b1, b2, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, eps, r.t)) {
    r.hit = __float_as_int(f.v3.w);
    if (ANY) return kDone;
  }
  if (cnt > 2) {
    r.ref = (int)(u + 2u - (2u << b.leaf_shift));
    return kContinue;
  }
  if (r.sp == 0) return kDone;
  r.ref = stack[--r.sp * stride];
  return kContinue;
}

// One step of a ray: an inner node or up to two triangles of a leaf.
template <bool ANY, bool FASTMM, bool LONE = false>
__device__ __forceinline__ StepResult ray_step(const DevBVH& b, RayState& r, float eps, int* stack, int stride,
                                               int limit) {
  Fetch f;
  fetch<LONE>(b, r.ref, f);
  if (r.ref < 0) return leaf_step<ANY>(b, f, r, eps, stack, stride);
  if (ANY) return inner_step_any<FASTMM>(b, f, r, stack, stride, limit);
  return FASTMM ? inner_step_sorted(f, r, stack, stride, limit) : inner_step(b, f, r, stack, stride, limit);
}

// Whole traversal of one ray by one thread. ANY = stop at the first hit
// (traverseMBVHShadow: nodes culled against maxDist, triangles accepted below
// it). `stack` is this thread's column of a [entries][stride] shared array.
// Returns false when the stack limit was reached (the ray's result is dropped).
template <bool ANY, bool FASTMM>
__device__ __forceinline__ bool traverse(const DevBVH& b, RayState& r, float eps, int* stack, int stride) {
  const int limit = b.stack_entries;
  while (true) {
    const StepResult s = ray_step<ANY, FASTMM>(b, r, eps, stack, stride, limit);
    if (s == kDone) return true;
    if (s == kOverflow) return false;
  }
}

// Persistent traversal with per-warp dynamic ray fetch. Each lane owns a ray
// and performs one step (an inner node or a leaf) per round; lanes whose ray
// finished take the next rays from a device cursor (one atomicAdd per warp),
// so a warp is not held back by its longest ray. A warp refills once at least
// REFILL of its lanes are idle (or all are): refilling costs a cursor atomic
// shared by every warp, a ballot and the new rays' loads and reciprocals, run
// by the whole warp for the lanes that refill, so batching refills pays for
// long incoherent traversals (the wavefront's extend) while short coherent
// queries refill at the first idle lane. Every ray still performs the
// reference's exact sequence of node tests, pushes, pops and triangle tests:
// only the interleaving across lanes changes.
//   IO::load(int i, float4& org, float4& dir, float& t0)
//   IO::store(int i, const RayState& r, bool overflow)
template <bool ANY, bool FASTMM, int REFILL, bool LONE, class IO>
__device__ __forceinline__ void trace_persistent(const DevBVH& b, int n, int* cursor, float eps, IO& io, int* stack,
                                                 int stride, int lanes = 32) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned own = FULL >> (32 - lanes);  // the lanes that take rays (lanes_for)
  const unsigned below = (1u << lane) - 1u;
  const int limit = b.stack_entries;
  int rid = -1;
  bool exhausted = false;
  RayState r;
  r.ref = kEmptyChild;
  while (true) {
    if (!exhausted) {
      const unsigned m = __ballot_sync(FULL, rid < 0) & own;
      if (m == own || __popc(m) >= REFILL) {
        const int leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(cursor, __popc(m));
        base = __shfl_sync(FULL, base, leader);
        if (base + __popc(m) >= n) exhausted = true;
        if (rid < 0 && lane < lanes) {
          const int my = base + __popc(m & below);
          if (my < n) {
            float4 o, d;
            float t0;
            io.load(my, o, d, t0);
            ray_begin(b, r, o, d, t0);
            rid = my;
          }
        }
      }
    }
    if (__ballot_sync(FULL, rid >= 0) == 0) break;
    if (rid < 0) continue;
    const StepResult s = ray_step<ANY, FASTMM, LONE>(b, r, eps, stack, stride, limit);
    if (s != kContinue) {
      io.store(rid, r, s == kOverflow);
      rid = -1;
    }
  }
}

// trace_persistent with a BVH and epsilon per lane: io.load(i, o, d, t0, b, eps)
// supplies the ray and the tree it is traced against (batches of jobs).
template <bool ANY, bool FASTMM, int REFILL, class IO>
__device__ __forceinline__ void trace_persistent_batch(int n, int* cursor, IO& io, int* stack, int stride, int lanes) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const unsigned own = FULL >> (32 - lanes);  // the lanes that take rays (batch_lanes)
  int rid = -1;
  bool exhausted = false;
  RayState r;
  r.ref = kEmptyChild;
  DevBVH b;
  float eps = 0.0f;
  while (true) {
    if (!exhausted) {
      const unsigned m = __ballot_sync(FULL, rid < 0) & own;
      if (m == own || __popc(m) >= REFILL) {
        const int leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(cursor, __popc(m));
        base = __shfl_sync(FULL, base, leader);
        if (base + __popc(m) >= n) exhausted = true;
        if (rid < 0 && lane < lanes) {
          const int my = base + __popc(m & below);
          if (my < n) {
            float4 o, d;
            float t0;
            io.load(my, o, d, t0, b, eps);
            ray_begin(b, r, o, d, t0);
            rid = my;
          }
        }
      }
    }
    if (__ballot_sync(FULL, rid >= 0) == 0) break;
    if (rid < 0) continue;
    const StepResult s = ray_step<ANY, FASTMM>(b, r, eps, stack, stride, b.stack_entries);
    if (s != kContinue) {
      io.store(rid, r, s == kOverflow);
      rid = -1;
    }
  }
}

}  // namespace ct

// Exact point-triangle closest point and the 4-wide BVH traversal (device).
//
// The triangle routine restates Ericson, Real-Time Collision Detection §5.1.5,
// in the operation order of the reference CPU oracle
// (src/geometry/closest_point.cpp:7-48, device twin src/cuda/bvh_query.cu:33-73).
// Every arithmetic step uses a round-to-nearest intrinsic (__fadd_rn etc.), which
// the compiler never fuses into an FMA, so results are bit-identical to the
// reference's g++ build of the same expressions.  The axis-aligned box distance
// uses the same non-fused operations, which keeps it a rounding-monotone lower
// bound of every contained triangle's computed distance; over the frame nodes
// prune_limit adds a margin for the frame's rounding.  Pruning therefore never
// drops a triangle whose distance ties the current best, and the (d2, id)
// tie-break returns the lowest triangle id among exact ties — the
// answer of the reference brute force, which keeps the first minimum in index
// order (closest_point.cpp:57-65).
#pragma once

#include <float.h>
#include <stdint.h>

#include "layout.h"

namespace n2w {
namespace dev {

struct V3 {
  float x, y, z;
};

__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return V3{fs(a.x, b.x), fs(a.y, b.y), fs(a.z, b.z)}; }
__device__ __forceinline__ V3 vadd(V3 a, V3 b) { return V3{fa(a.x, b.x), fa(a.y, b.y), fa(a.z, b.z)}; }
__device__ __forceinline__ V3 vscale(V3 a, float s) { return V3{fm(a.x, s), fm(a.y, s), fm(a.z, s)}; }
__device__ __forceinline__ float vdot(V3 a, V3 b) { return fa(fa(fm(a.x, b.x), fm(a.y, b.y)), fm(a.z, b.z)); }

// Ericson closest point on triangle abc to p, reference operation order.
// Branch-free form for SIMT: all six dot products and the three barycentric
// numerators are computed, the Voronoi region is chosen with Ericson's tests in
// his order, and only the chosen region's expression is evaluated (one IEEE
// division); each region's result uses exactly the reference's operations:
//   edge ab: a + ab*(d1/(d1-d3))           edge ac: a + ac*(d2/(d2-d6))
//   edge bc: b + (c-b)*((d4-d3)/((d4-d3)+(d5-d6)))
//   face:    (a + ab*(vb*r)) + ac*(vc*r),  r = 1/((va+vb)+vc)
//   vertex regions return the vertex itself.
// The edges ab = b - a and ac = c - a come with the triangle (TriEdges).
__device__ __forceinline__ V3 closest_point_triangle(V3 p, V3 a, V3 b, V3 c, V3 ab, V3 ac) {
  const V3 ap = vsub(p, a);
  const float d1 = vdot(ab, ap);
  const float d2 = vdot(ac, ap);
  const V3 bp = vsub(p, b);
  const float d3 = vdot(ab, bp);
  const float d4 = vdot(ac, bp);
  const V3 cq = vsub(p, c);
  const float d5 = vdot(ab, cq);
  const float d6 = vdot(ac, cq);
  const float vc = fs(fm(d1, d4), fm(d3, d2));
  const float vb = fs(fm(d5, d2), fm(d1, d6));
  const float va = fs(fm(d3, d6), fm(d5, d4));
  const float d43 = fs(d4, d3);
  const float d56 = fs(d5, d6);

  const bool rA = d1 <= 0.0f && d2 <= 0.0f;
  const bool rB = !rA && d3 >= 0.0f && d4 <= d3;
  const bool rAB = !rA && !rB && vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f;
  const bool r3 = rA || rB || rAB;
  const bool rC = !r3 && d6 >= 0.0f && d5 <= d6;
  const bool rAC = !r3 && !rC && vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f;
  const bool rBC = !r3 && !rC && !rAC && va <= 0.0f && d43 >= 0.0f && d56 >= 0.0f;
  const bool rF = !r3 && !rC && !rAC && !rBC;

  float num = 0.0f, den = 1.0f;
  if (rAB) { num = d1; den = fs(d1, d3); }
  if (rAC) { num = d2; den = fs(d2, d6); }
  if (rBC) { num = d43; den = fa(d43, d56); }
  if (rF) { num = 1.0f; den = fa(fa(va, vb), vc); }
  const float q = fd(num, den);
  const float s = rF ? fm(vb, q) : q;
  const V3 base = rBC ? b : a;
  const V3 e1 = rBC ? vsub(c, b) : (rAC ? ac : ab);
  V3 r = vadd(base, vscale(e1, s));
  if (rF) r = vadd(r, vscale(ac, fm(vc, q)));
  if (rA) r = a;
  if (rB) r = b;
  if (rC) r = c;
  return r;
}

// Signed gap from p to [lo, hi] along one axis: p - clamp(p, lo, hi).  Its
// square equals that of max(lo - p, p - hi, 0) bit for bit (IEEE subtraction
// is sign-symmetric), with one subtraction instead of two; empty slots
// (lo = +inf, hi = -inf) give an infinite gap.
__device__ __forceinline__ float axis_gap(float p, float lo, float hi) {
  return fs(p, fminf(fmaxf(p, lo), hi));
}

__device__ __forceinline__ float box_d2(V3 p, float lox, float hix, float loy, float hiy, float loz,
                                        float hiz) {
  const float dx = axis_gap(p.x, lox, hix);
  const float dy = axis_gap(p.y, loy, hiy);
  const float dz = axis_gap(p.z, loz, hiz);
  return fa(fa(fm(dx, dx), fm(dy, dy)), fm(dz, dz));
}

// ---- contracted-FP32 variants for the walker -------------------------------
// A walk only needs each step's distance (and the closest point at the
// terminal step) to FP32 accuracy: the reference's GPU walker is compiled
// with FMA contraction and IEEE division, and its parity with any CPU
// evaluation is statistical.  These variants evaluate the same Ericson region
// tests with fused multiply-adds and the fast division intrinsic, cutting the
// instruction count of a triangle test by about a quarter.  Results differ
// from the exact routine above by a few ulps, so the walker's queries are not
// bit-identical to n2w_bvh_query_device's; the query API keeps the exact path.
__device__ __forceinline__ float vdot_fast(V3 a, V3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ V3 vsub_fast(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 vmad_fast(V3 e, float s, V3 base) {
  return V3{fmaf(e.x, s, base.x), fmaf(e.y, s, base.y), fmaf(e.z, s, base.z)};
}

__device__ __forceinline__ V3 closest_point_triangle_fast(V3 p, V3 a, V3 b, V3 c, V3 ab, V3 ac) {
  const V3 ap = vsub_fast(p, a);
  const float d1 = vdot_fast(ab, ap);
  const float d2 = vdot_fast(ac, ap);
  const V3 bp = vsub_fast(p, b);
  const float d3 = vdot_fast(ab, bp);
  const float d4 = vdot_fast(ac, bp);
  const V3 cq = vsub_fast(p, c);
  const float d5 = vdot_fast(ab, cq);
  const float d6 = vdot_fast(ac, cq);
  const float vc = fmaf(d1, d4, -(d3 * d2));
  const float vb = fmaf(d5, d2, -(d1 * d6));
  const float va = fmaf(d3, d6, -(d5 * d4));
  const float d43 = d4 - d3;
  const float d56 = d5 - d6;

  const bool rA = d1 <= 0.0f && d2 <= 0.0f;
  const bool rB = !rA && d3 >= 0.0f && d4 <= d3;
  const bool rAB = !rA && !rB && vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f;
  const bool r3 = rA || rB || rAB;
  const bool rC = !r3 && d6 >= 0.0f && d5 <= d6;
  const bool rAC = !r3 && !rC && vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f;
  const bool rBC = !r3 && !rC && !rAC && va <= 0.0f && d43 >= 0.0f && d56 >= 0.0f;
  const bool rF = !r3 && !rC && !rAC && !rBC;

  float num = 0.0f, den = 1.0f;
  if (rAB) { num = d1; den = d1 - d3; }
  if (rAC) { num = d2; den = d2 - d6; }
  if (rBC) { num = d43; den = d43 + d56; }
  if (rF) { num = 1.0f; den = (va + vb) + vc; }
  const float q = __fdividef(num, den);
  const float s = rF ? vb * q : q;
  const V3 base = rBC ? b : a;
  const V3 e1 = rBC ? vsub_fast(c, b) : (rAC ? ac : ab);
  V3 r = vmad_fast(e1, s, base);
  if (rF) r = vmad_fast(ac, vc * q, r);
  if (rA) r = a;
  if (rB) r = b;
  if (rC) r = c;
  return r;
}

__device__ __forceinline__ void cswap(float& da, int& ra, float& db, int& rb) {
  if (db < da) {
    const float td = da;
    da = db;
    db = td;
    const int tr = ra;
    ra = rb;
    rb = tr;
  }
}

// One 4-wide node (layout.h Node4: lo_x, hi_x, lo_y, hi_y, lo_z, hi_z float4,
// then the child refs) in four 256-bit read-only loads (ld.global.nc.v8,
// sm_100) instead of seven 128-bit ones: a warp's divergent gathers touch
// the same sectors with fewer L1 wavefronts.  Node arrays are cudaMalloc'd
// (256-byte aligned) and nodes are 128 bytes, so every load is 32-byte
// aligned.  The last load also brings the node's 16 pad bytes (same sector).
// The loads do not allocate in L1: a quarter of them hit there, and filling
// lines for the rest took the data pipe (75 % busy) that serves the hits and
// the lanes' lists.  262,144 / 4,194,304 uniform queries 391 -> 374 us / 4.77 ->
// 4.37 ms, Laplace / Poisson walks 17.4 -> 16.0 / 46.1 -> 43.4 ms, batched
// instances 37.3 -> 33.8 ms (evict_first: 17.1 / 45.0 / 36.4; evict_last: as
// without a hint).  kL1 keeps the allocation where most loads do hit: launches of
// few walkers per SM, small trees (fits_l1) and the axis-aligned boxes.
template <bool kL1 = false>
__device__ __forceinline__ void ldg_v8f(const float4* p, float4& a, float4& b) {
  if constexpr (kL1) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
  } else {
    asm("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
  }
}
__device__ __forceinline__ int4 ldg_v8_first_int4(const float4* p) {
  int4 a;
  int d0, d1, d2, d3;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3)
      : "l"(p));
  return a;
}
template <bool kL1>
__device__ __forceinline__ void load_node(const float4* __restrict__ nodes, int32_t ref, float4& lox, float4& hix,
                                          float4& loy, float4& hiy, float4& loz, float4& hiz, int4& ch) {
  static_assert(sizeof(Node4) == 128, "node loads assume 128-byte nodes");
  const float4* n = nodes + static_cast<size_t>(ref) * 8;
  ldg_v8f<kL1>(n + 0, lox, hix);
  ldg_v8f<kL1>(n + 2, loy, hiy);
  ldg_v8f<kL1>(n + 4, loz, hiz);
  ch = ldg_v8_first_int4(n + 6);
}

// Squared distances from p to the four child boxes of an axis-aligned node; returns
// its child references.
template <bool kL1 = false>
__device__ __forceinline__ int4 box_distances(const float4* __restrict__ nodes, int32_t ref, V3 p, float (&d)[4]) {
  float4 lox, hix, loy, hiy, loz, hiz;
  int4 ch;
  load_node<kL1>(nodes, ref, lox, hix, loy, hiy, loz, hiz, ch);
  d[0] = box_d2(p, lox.x, hix.x, loy.x, hiy.x, loz.x, hiz.x);
  d[1] = box_d2(p, lox.y, hix.y, loy.y, hiy.y, loz.y, hiz.y);
  d[2] = box_d2(p, lox.z, hix.z, loy.z, hiy.z, loz.z, hiz.z);
  d[3] = box_d2(p, lox.w, hix.w, loy.w, hiy.w, loz.w, hiz.w);
  return ch;
}

struct Rec64 {  // a 64-byte record as loaded
  float4 r0, r1, r2, r3;
};
template <bool kL1>
__device__ __forceinline__ Rec64 load_rec(const float4* __restrict__ base, int index) {
  const float4* t = base + static_cast<size_t>(index) * 4;
  Rec64 r;
  ldg_v8f<kL1>(t + 0, r.r0, r.r1);
  ldg_v8f<kL1>(t + 2, r.r2, r.r3);
  return r;
}

// ---- frame nodes (layout.h FrameNode4) ------------------------------------------
// The mirror of a node's frame; v.z from |v|^2 = 2 (off by at most 2^-22 v.z).
__device__ __forceinline__ V3 frame_v(float x, float y) {
  float z;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(z) : "f"(fmaxf(fmaf(-x, x, fmaf(-y, y, 2.0f)), 0.0f)));
  return v3(x, y, z);
}

// p in the frame: p - v (v.p).
__device__ __forceinline__ V3 to_frame(V3 v, V3 p) {
  const float s = fmaf(v.z, p.z, fmaf(v.y, p.y, v.x * p.x));
  return V3{fmaf(-s, v.x, p.x), fmaf(-s, v.y, p.y), fmaf(-s, v.z, p.z)};
}

struct FrameData {
  V3 v, o;
  float step[3];      // 2^e of each axis
  uint32_t plane[6];
  int4 ch;
};
__device__ __forceinline__ FrameData decode_frame_node(const Rec64& r) {
  const float4 a = r.r0, b = r.r1, c = r.r2, d = r.r3;
  FrameData f;
  f.v = frame_v(a.x, a.y);
  f.o = v3(a.z, a.w, b.x);
  const uint32_t e = __float_as_uint(b.y);
  f.step[0] = __uint_as_float((e << 23) & 0x7f800000u);
  f.step[1] = __uint_as_float((e << 15) & 0x7f800000u);
  f.step[2] = __uint_as_float((e << 7) & 0x7f800000u);
  f.plane[0] = __float_as_uint(b.z);
  f.plane[1] = __float_as_uint(b.w);
  f.plane[2] = __float_as_uint(c.x);
  f.plane[3] = __float_as_uint(c.y);
  f.plane[4] = __float_as_uint(c.z);
  f.plane[5] = __float_as_uint(c.w);
  f.ch = make_int4(__float_as_int(d.x), __float_as_int(d.y), __float_as_int(d.z), __float_as_int(d.w));
  return f;
}

template <bool kL1 = false>
__device__ __forceinline__ FrameData load_frame_node(const float4* __restrict__ frames, int32_t ref) {
  return decode_frame_node(load_rec<kL1>(frames, ref));
}

// 32768 + byte k of w: the byte's bits in the mantissa.
template <int k>
__device__ __forceinline__ float plane_bits(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7404u + (k << 4)));
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// The largest of a, b and 0; NaN if one is.
__device__ __forceinline__ float max3_0(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, 0f00000000;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Adds one axis's squared gaps between q (relative to o) and the boxes of
// children k, k + 1: max(lo - q, q - hi, 0) with the planes (32768 + b) 2^e -
// 32768 2^e folded into the subtractions (near = -32768 2^e - q, rounded by at
// most 2^-9 of a step or u |q|; far = -near).
template <int k>
__device__ __forceinline__ uint64_t add_gap2(uint64_t d, uint32_t wlo, uint32_t whi, uint64_t step, uint64_t neg_step,
                                             uint64_t near, uint64_t far) {
  float l0, l1, h0, h1;
  unpack2(fma2(pack2(plane_bits<k>(wlo), plane_bits<k + 1>(wlo)), step, near), l0, l1);
  unpack2(fma2(pack2(plane_bits<k>(whi), plane_bits<k + 1>(whi)), neg_step, far), h0, h1);
  const uint64_t g = pack2(max3_0(l0, h0), max3_0(l1, h1));
  return fma2(g, g, d);
}

// Squared distances from p to the four child boxes of a node (two children per
// instruction where there is a packed form; slots without a child: any number).
__device__ __forceinline__ void frame_distances(const FrameData& f, V3 p, float (&d)[4]) {
  const V3 m = to_frame(f.v, p);
  const float q[3] = {m.x - f.o.x, m.y - f.o.y, m.z - f.o.z};
  uint64_t d01 = 0, d23 = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float s = f.step[a], nr = fmaf(-32768.0f, s, -q[a]);
    const uint64_t step = pack2(s, s), neg_step = pack2(-s, -s), near = pack2(nr, nr), far = pack2(-nr, -nr);
    d01 = add_gap2<0>(d01, f.plane[2 * a], f.plane[2 * a + 1], step, neg_step, near, far);
    d23 = add_gap2<2>(d23, f.plane[2 * a], f.plane[2 * a + 1], step, neg_step, near, far);
  }
  unpack2(d01, d[0], d[1]);
  unpack2(d23, d[2], d[3]);
}

__device__ __forceinline__ bool is_leaf(int c) { return static_cast<int>(0u - static_cast<unsigned>(c)) > 0; }

// Largest computed box distance^2, in a node's frame, that a box holding a
// triangle at computed distance^2 `best` can have.  With u = 2^-24 the frame's
// coordinates of p are off by at most 8 u |p|, |v|^2 by 12 u and the distance
// and its square by a few u more; the boxes carry the triangles' own rounding
// (build_frames).  2^-20 |p|_1 = 16 u |p|_1 and a factor 1 + 2^-17 cover these
// twice over, so no triangle that ties the best distance is pruned.
__device__ __forceinline__ float prune_limit(float best, V3 p) {
  float s;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(best));
  s = fmaf(fabsf(p.x) + fabsf(p.y) + fabsf(p.z), 9.5367431640625e-07f, s);
  return fminf(s * s * 1.00000762939453125f, FLT_MAX);
}

struct ClosestHit {
  float d2;
  float lim;  // prune_limit of d2 (traversals over frame nodes)
  int id;    // original triangle id; INT32_MAX when nothing was found below the bound
  int slot;  // leaf-order index of that triangle (used to re-seed the next query)
  V3 cp;
};

// Tests one triangle (by leaf-order slot) and keeps it if it beats the hit in
// (d2, id) order.  Seeding a query with real candidates gives the traversal a
// tight bound without changing its answer.  kFast selects the contracted-FP32
// triangle routine (walker); callers use the test_slot / test_slot_fast wrappers.
template <bool kFast>
__device__ __forceinline__ void test_rec(const Rec64& rec, int slot, V3 p, ClosestHit& hit) {
  const float4 r0 = rec.r0, r1 = rec.r1, r2 = rec.r2, r3 = rec.r3;
  const V3 a = v3(r0.x, r0.y, r0.z), ab = v3(r1.x, r1.y, r1.z), ac = v3(r1.w, r2.x, r2.y),
           b = v3(r2.z, r2.w, r3.x), c = v3(r3.y, r3.z, r3.w);
  V3 cp;
  float dd;
  if (kFast) {
    cp = closest_point_triangle_fast(p, a, b, c, ab, ac);
    const V3 dv = vsub_fast(cp, p);
    dd = vdot_fast(dv, dv);
  } else {
    cp = closest_point_triangle(p, a, b, c, ab, ac);
    const V3 dv = vsub(cp, p);
    dd = vdot(dv, dv);
  }
  const int id = __float_as_int(r0.w);
  if (dd < hit.d2 || (dd == hit.d2 && id < hit.id)) {
    hit.d2 = dd;
    hit.lim = prune_limit(dd, p);
    hit.id = id;
    hit.slot = slot;
    hit.cp = cp;
  }
}

template <bool kFast, bool kL1 = false>
__device__ __forceinline__ void test_slot_impl(const float4* __restrict__ tris, int slot, V3 p, ClosestHit& hit) {
  test_rec<kFast>(load_rec<kL1>(tris, slot), slot, p, hit);
}
template <bool kL1 = false>
__device__ __forceinline__ void test_slot(const float4* __restrict__ tris, int slot, V3 p, ClosestHit& hit) {
  test_slot_impl<false, kL1>(tris, slot, p, hit);
}
template <bool kL1>
__device__ __forceinline__ void test_slot_fast(const float4* __restrict__ tris, int slot, V3 p, ClosestHit& hit) {
  test_slot_impl<true, kL1>(tris, slot, p, hit);
}

// Seed grid: (n+1)^3 lattice nodes over a padded mesh box.  A node's cell {x: the
// leaf slot of the triangle closest to the node; y, z, w: up to kCellEntries
// subtrees (child references, kEmptyChild when unused) that hold the closest
// triangle of every point nearer to this lattice node than to any other}.  The
// triangle is a candidate within (node distance + |x - node|) of x; starting at
// the subtrees instead of the root skips the top of the tree.
constexpr int kCellEntries = 3;
struct SeedGrid {
  const int4* cells;  // nullptr when absent
  float lo_x, lo_y, lo_z;
  float inv_h;
  int n;      // cells per axis
  float far;  // distance from the lattice's centre, in half lattices, from which queries search boxes (far_limit)
};

// The cell of the lattice node nearest to p; outside the lattice the clamped
// node's cell with the root as its only subtree.  (Walks stay inside; the counted
// query's seeds, which the CPU restatement reproduces.)
__device__ __forceinline__ int4 seed_cell(const SeedGrid& g, V3 p, int root) {
  const float fx = (p.x - g.lo_x) * g.inv_h, fy = (p.y - g.lo_y) * g.inv_h, fz = (p.z - g.lo_z) * g.inv_h;
  const float n = static_cast<float>(g.n);
  const float cx = fminf(fmaxf(fx, 0.0f), n), cy = fminf(fmaxf(fy, 0.0f), n), cz = fminf(fmaxf(fz, 0.0f), n);
  const int s = g.n + 1;
  int4 c = __ldg(g.cells + (static_cast<size_t>(__float2int_rn(cz)) * s + __float2int_rn(cy)) * s + __float2int_rn(cx));
  if (!(cx == fx && cy == fy && cz == fz)) {
    c.y = root;
    c.z = c.w = kEmptyChild;
  }
  return c;
}

// The same for any point: outside the lattice the cell where the ray from the
// lattice's centre to p leaves it, with the root as its only subtree.  (A point
// clamped axis by axis lies in another direction from the mesh, and its triangle is
// a poor seed.)  300,000 queries around 81,920 triangles, 5 extents from their centre:
// 3,535 -> 869 us, 1.5 extents: 2,017 -> 645 us.  `far`: the margin of the frame nodes'
// limit at p is large against the triangles (far_limit).
__device__ __forceinline__ int4 seed_cell_any(const SeedGrid& g, V3 p, int root, bool& far) {
  const float fx = (p.x - g.lo_x) * g.inv_h, fy = (p.y - g.lo_y) * g.inv_h, fz = (p.z - g.lo_z) * g.inv_h;
  const float n = static_cast<float>(g.n), half = 0.5f * n;
  float cx = fminf(fmaxf(fx, 0.0f), n), cy = fminf(fmaxf(fy, 0.0f), n), cz = fminf(fmaxf(fz, 0.0f), n);
  const bool in = cx == fx && cy == fy && cz == fz;
  far = false;
  if (!in) {
    const float dx = fx - half, dy = fy - half, dz = fz - half;
    const float out = fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)));
    const float s = half / out;
    cx = fminf(fmaxf(fmaf(dx, s, half), 0.0f), n);  // (not a number: node 0)
    cy = fminf(fmaxf(fmaf(dy, s, half), 0.0f), n);
    cz = fminf(fmaxf(fmaf(dz, s, half), 0.0f), n);
    far = out > half * g.far;
  }
  const int m = g.n + 1;
  int4 c = __ldg(g.cells + (static_cast<size_t>(__float2int_rn(cz)) * m + __float2int_rn(cy)) * m + __float2int_rn(cx));
  if (!in) {
    c.y = root;
    c.z = c.w = kEmptyChild;
  }
  return c;
}

// A tree as queries search it.  The arrays share node indices and leaves, and the
// answer is the same over either.
struct QueryNodes {
  const float4* frames;  // FrameNode4
  const float4* boxes;   // Node4
  bool use_boxes;        // the tree's choice (choose_nodes)
  // The seed cell of p: where boxes fit, the clamped node is closer to the answer than the
  // one on the ray (1,000 queries around an axis-aligned cube: 14 us against 60).
  __device__ __forceinline__ int4 seed(const SeedGrid& g, V3 p, int root, bool& far) const {
    far = false;
    return use_boxes ? seed_cell(g, p, root) : seed_cell_any(g, p, root, far);
  }
};

struct TraversalStats {
  int node_visits;
  int tri_tests;
  int overflow;
};

// Ordered depth-first traversal: at each inner node the four child boxes are
// measured, sorted ascending (fixed 5-comparator network), the nearest child
// is entered and the others are pushed far-to-near.  Popped entries are
// re-checked against the current best.  Candidates are any triangles whose box
// distance is <= best_d2; `hit` must be initialised by the caller (cold query:
// d2 = FLT_MAX, id = INT32_MAX; warm start: d2 = an upper bound).
__device__ __forceinline__ void traverse(const float4* __restrict__ nodes,
                                         const float4* __restrict__ tris, V3 p, ClosestHit& hit,
                                         TraversalStats& st, int32_t root = 0) {
  int2 stack[kTraversalStack];
  int sp = 0;
  int32_t ref = root;
  for (;;) {
    if (ref >= 0) {
      ++st.node_visits;
      const float4* n = nodes + static_cast<size_t>(ref) * 8;
      const float4 lox = __ldg(n + 0);
      const float4 hix = __ldg(n + 1);
      const float4 loy = __ldg(n + 2);
      const float4 hiy = __ldg(n + 3);
      const float4 loz = __ldg(n + 4);
      const float4 hiz = __ldg(n + 5);
      const int4 ch = __ldg(reinterpret_cast<const int4*>(n + 6));
      float d0 = box_d2(p, lox.x, hix.x, loy.x, hiy.x, loz.x, hiz.x);
      float d1 = box_d2(p, lox.y, hix.y, loy.y, hiy.y, loz.y, hiz.y);
      float d2 = box_d2(p, lox.z, hix.z, loy.z, hiy.z, loz.z, hiz.z);
      float d3 = box_d2(p, lox.w, hix.w, loy.w, hiy.w, loz.w, hiz.w);
      int r0 = ch.x, r1 = ch.y, r2 = ch.z, r3 = ch.w;
      cswap(d0, r0, d1, r1);
      cswap(d2, r2, d3, r3);
      cswap(d0, r0, d2, r2);
      cswap(d1, r1, d3, r3);
      cswap(d1, r1, d2, r2);
      const float best = hit.d2;
      if (d3 <= best) {
        if (sp < kTraversalStack) stack[sp++] = make_int2(r3, __float_as_int(d3));
        else st.overflow = 1;
      }
      if (d2 <= best) {
        if (sp < kTraversalStack) stack[sp++] = make_int2(r2, __float_as_int(d2));
        else st.overflow = 1;
      }
      if (d1 <= best) {
        if (sp < kTraversalStack) stack[sp++] = make_int2(r1, __float_as_int(d1));
        else st.overflow = 1;
      }
      ref = (d0 <= best) ? r0 : kEmptyChild;
    } else if (ref != kEmptyChild) {
      const int first = leaf_first(ref);
      const int count = leaf_count(ref);
      st.tri_tests += count;
      for (int i = 0; i < count; ++i) test_slot_impl<false>(tris, first + i, p, hit);
      ref = kEmptyChild;
    }
    if (ref == kEmptyChild) {
      bool found = false;
      while (sp > 0) {
        const int2 e = stack[--sp];
        if (__int_as_float(e.y) <= hit.d2) {
          ref = e.x;
          found = true;
          break;
        }
      }
      if (!found) break;
    }
  }
}

// ---- one lane's query over the axis-aligned nodes, unit by unit ----------------
// (the counted query, whose visit counts the CPU restatement reproduces, and the
// trees whose frames do not pay)
struct TravState {
  int sp;
  int ref;       // inner node to expand next, or kEmptyChild
  int leaf_cur;  // next triangle slot of the leaf being tested
  int leaf_end;
};

// One unit of traversal work: test ONE triangle of the current leaf, or expand
// ONE 4-wide node (same ordering and pruning as dev::traverse: children sorted
// by box distance, nearest entered, others pushed far-to-near, popped entries
// re-checked).  Returns false once the query is complete.
template <bool kL1>
__device__ __forceinline__ bool trav_step_boxes(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                                V3 p, ClosestHit& hit, TravState& t, int2* stack, uint32_t& c_nodes,
                                                uint32_t& c_tris, bool& overflow) {
  if (t.leaf_cur >= t.leaf_end && t.ref == kEmptyChild) {
    bool found = false;
    while (t.sp > 0) {
      const int2 e = stack[--t.sp];
      if (__int_as_float(e.y) <= hit.d2) {
        if (e.x >= 0) {
          t.ref = e.x;
        } else {
          t.leaf_cur = leaf_first(e.x);
          t.leaf_end = t.leaf_cur + leaf_count(e.x);
        }
        found = true;
        break;
      }
    }
    if (!found) return false;
  }
  if (t.leaf_cur < t.leaf_end) {
    test_slot_impl<false, kL1>(tris, t.leaf_cur, p, hit);
    ++t.leaf_cur;
    ++c_tris;
    return true;
  }
  float d[4];
  const int4 ch = box_distances<kL1>(nodes, t.ref, p, d);
  ++c_nodes;
  float d0 = d[0], d1 = d[1], d2 = d[2], d3 = d[3];
  int r0 = ch.x, r1 = ch.y, r2 = ch.z, r3 = ch.w;
  cswap(d0, r0, d1, r1);
  cswap(d2, r2, d3, r3);
  cswap(d0, r0, d2, r2);
  cswap(d1, r1, d3, r3);
  cswap(d1, r1, d2, r2);
  const float best = hit.d2;
  auto push = [&](float d, int r) {
    if (d <= best) {
      if (t.sp < kTraversalStack) stack[t.sp++] = make_int2(r, __float_as_int(d));
      else overflow = true;
    }
  };
  push(d3, r3);
  push(d2, r2);
  push(d1, r1);
  t.ref = kEmptyChild;
  if (d0 <= best) {
    if (r0 >= 0) {
      t.ref = r0;
    } else {
      t.leaf_cur = leaf_first(r0);
      t.leaf_end = t.leaf_cur + leaf_count(r0);
    }
  }
  return true;
}

// ---- one lane's query over the frame nodes, advanced in steps -------------------
// A query keeps two lists, inner nodes to expand and leaves to test, and a step
// takes one triangle from the one and one node from the other.  A warp runs
// both code paths in every iteration anyway (its lanes are never all at the
// same kind of work), so a lane that has both kinds pending advances in both:
// 16.7 iterations per walk query for 14.2 expansions and 8.1 tests, against
// 22.3 one by one.  A walk's query is seeded with triangles close to the answer,
// so its order hardly matters: children are neither sorted nor re-checked when
// they are taken up (+0.2 % expansions, +7 % tests along walks), and an entry
// is its 4-byte reference.  (8-byte entries with distances, sorted and re-checked,
// cost exact queries of smooth meshes 12-15 %.)  Nodes wait while more than kLeafRoom leaves are
// pending, which bounds the leaf list.
constexpr int kLeafStack = 16;
constexpr int kLeafRoom = kLeafStack - 4;  // a node adds at most four leaves

struct FrameTrav {
  int np, lp;              // entries on the two lists
  int ref;                 // inner node to expand next, or kEmptyChild
  int leaf_cur, leaf_end;  // triangle slots of the leaf being tested
  __device__ __forceinline__ void start(int root) {
    np = lp = 0;
    ref = root;
    leaf_cur = leaf_end = 0;
  }
  // Starts at the subtrees of a seed cell (seed_cell).
  template <class Stack>
  __device__ __forceinline__ void start(int4 cell, Stack& st) {
    start(kEmptyChild);
    enter(cell.y, st);
    enter(cell.z, st);
    enter(cell.w, st);
  }
  template <class Stack>
  __device__ __forceinline__ void enter(int e, Stack& st) {
    if (e >= 0) {
      if (ref != kEmptyChild) st.nodes[np++] = ref;
      ref = e;
    } else if (e != kEmptyChild) {
      st.leaves[lp++] = e;
    }
  }
  __device__ __forceinline__ bool done() const {
    return ref == kEmptyChild && leaf_cur >= leaf_end && np == 0 && lp == 0;
  }
};
struct FrameStack {
  int nodes[kTraversalStack + 3];
  int leaves[kLeafStack];
};

// Tests one pending triangle, if there is one.  The current best is not tested
// again (queries start with it tested as a seed).
template <bool kFast, bool kL1 = false>
__device__ __forceinline__ void trav_triangle(const float4* __restrict__ tris, V3 p, ClosestHit& hit, FrameTrav& t,
                                              FrameStack& st, uint32_t& c_tris) {
  if (t.leaf_cur >= t.leaf_end && t.lp > 0) {
    const int e = st.leaves[--t.lp];
    t.leaf_cur = leaf_first(e);
    t.leaf_end = t.leaf_cur + leaf_count(e);
  }
  if (t.leaf_cur < t.leaf_end) {
    if (t.leaf_cur != hit.slot) {
      test_slot_impl<kFast, kL1>(tris, t.leaf_cur, p, hit);
      ++c_tris;
    }
    ++t.leaf_cur;
  }
}

// Adds the children of a node that are within the limit to the lists, by predicated
// stores (branches per child left 9 of 32 lanes active); the last inner one is
// entered.  kNearest: the nearest child is moved to the last place.  Exact queries do
// this: their seeds can be poor (outside the lattice, on either side of a medial
// plane), and then the order decides how soon the limit tightens.  100,003 queries
// inside an axis-aligned cube of 120,000 triangles 118 -> 90 us, at its centre 378 ->
// 209, 5 extents from a torus of 80,000 634 -> 350; smooth closed meshes +-2 %.
template <bool kNearest>
__device__ __forceinline__ void expand_node(const Rec64& rec, V3 p, const ClosestHit& hit, FrameTrav& t, FrameStack& st,
                                            bool& overflow) {
  const FrameData f = decode_frame_node(rec);
  float d[4];
  frame_distances(f, p, d);
  int4 ch = f.ch;
  if constexpr (kNearest) {
    cswap(d[1], ch.y, d[0], ch.x);
    cswap(d[2], ch.z, d[1], ch.y);
    cswap(d[3], ch.w, d[2], ch.z);
  }
  const bool k0 = d[0] <= hit.lim, k1 = d[1] <= hit.lim, k2 = d[2] <= hit.lim, k3 = d[3] <= hit.lim;
  const bool n0 = k0 && ch.x >= 0, n1 = k1 && ch.y >= 0, n2 = k2 && ch.z >= 0, n3 = k3 && ch.w >= 0;
  const bool l0 = k0 && is_leaf(ch.x), l1 = k1 && is_leaf(ch.y), l2 = k2 && is_leaf(ch.z), l3 = k3 && is_leaf(ch.w);
  if (l0) st.leaves[t.lp] = ch.x;
  t.lp += l0 ? 1 : 0;
  if (l1) st.leaves[t.lp] = ch.y;
  t.lp += l1 ? 1 : 0;
  if (l2) st.leaves[t.lp] = ch.z;
  t.lp += l2 ? 1 : 0;
  if (l3) st.leaves[t.lp] = ch.w;
  t.lp += l3 ? 1 : 0;
  const bool p2 = n2 && n3, p1 = n1 && (n2 || n3), p0 = n0 && (n1 || n2 || n3);
  t.ref = n3 ? ch.w : (n2 ? ch.z : (n1 ? ch.y : (n0 ? ch.x : kEmptyChild)));
  if (p0) st.nodes[t.np] = ch.x;
  t.np += p0 ? 1 : 0;
  if (p1) st.nodes[t.np] = ch.y;
  t.np += p1 ? 1 : 0;
  if (p2) st.nodes[t.np] = ch.z;
  t.np += p2 ? 1 : 0;
  if (t.np > kTraversalStack) {  // the array holds three more than the limit
    t.np = kTraversalStack;
    overflow = true;
  }
}

// Expands one pending node, if there is one and the leaf list has room.
template <bool kL1 = false, bool kNearest = false>
__device__ __forceinline__ void trav_node(const float4* __restrict__ frames, V3 p, const ClosestHit& hit, FrameTrav& t,
                                          FrameStack& st, uint32_t& c_nodes, bool& overflow) {
  if (t.ref == kEmptyChild && t.np > 0) t.ref = st.nodes[--t.np];
  if (t.ref != kEmptyChild && t.lp <= kLeafRoom) {
    ++c_nodes;
    expand_node<kNearest>(load_rec<kL1>(frames, t.ref), p, hit, t, st, overflow);
  }
}

// trav_triangle and trav_node with both records loaded before either is used:
// one memory latency per step, for launches of so few walks that registers are
// plentiful and latency is all there is.
template <bool kFast, bool kL1>
__device__ __forceinline__ void trav_both(const float4* __restrict__ frames, const float4* __restrict__ tris, V3 p,
                                          ClosestHit& hit, FrameTrav& t, FrameStack& st, uint32_t& c_nodes,
                                          uint32_t& c_tris, bool& overflow) {
  if (t.leaf_cur >= t.leaf_end && t.lp > 0) {
    const int e = st.leaves[--t.lp];
    t.leaf_cur = leaf_first(e);
    t.leaf_end = t.leaf_cur + leaf_count(e);
  }
  if (t.ref == kEmptyChild && t.np > 0) t.ref = st.nodes[--t.np];
  const bool has_node = t.ref != kEmptyChild && t.lp <= kLeafRoom;
  bool has_tri = t.leaf_cur < t.leaf_end;
  const int slot = t.leaf_cur;
  if (has_tri) {
    ++t.leaf_cur;
    has_tri = slot != hit.slot;
  }
  Rec64 tri, node;
  if (has_tri) tri = load_rec<kL1>(tris, slot);
  if (has_node) node = load_rec<kL1>(frames, t.ref);
  if (has_tri) {
    test_rec<kFast>(tri, slot, p, hit);
    ++c_tris;
  }
  if (has_node) {
    ++c_nodes;
    expand_node<false>(node, p, hit, t, st, overflow);
  }
}

// A whole query in one lane (exact routines), seeded by the grid if there is one.
__device__ __forceinline__ void traverse_query(const QueryNodes& nodes, const float4* __restrict__ tris,
                                               const SeedGrid& grid, V3 p, ClosestHit& hit, TraversalStats& st,
                                               int32_t root) {
  const float4* __restrict__ frames = nodes.frames;
  FrameStack stack;
  FrameTrav t;
  if (grid.cells) {
    bool far;
    const int4 cell = nodes.seed(grid, p, root, far);
    test_slot(tris, cell.x, p, hit);
    ++st.tri_tests;
    if (nodes.use_boxes || far) {
      traverse(nodes.boxes, tris, p, hit, st, root);
      return;
    }
    t.start(cell, stack);
  } else {
    t.start(root);
  }
  uint32_t c_nodes = 0, c_tris = 0;
  bool overflow = false;
  while (!t.done()) {
    trav_triangle<false>(tris, p, hit, t, stack, c_tris);
    trav_node<false, true>(frames, p, hit, t, stack, c_nodes, overflow);
  }
  st.node_visits += static_cast<int>(c_nodes);
  st.tri_tests += static_cast<int>(c_tris);
  if (overflow) st.overflow = 1;
}

// +x ray / triangle test of the reference's slice mask
// (src/cuda/cubql_bvh.cu:407-428, Möller–Trumbore with its tolerances), in the
// same non-fused float operations, so the parity count matches the CPU test.
__device__ __forceinline__ bool ray_x_hits(V3 p, V3 a, V3 b, V3 c) {
  const float y_min = fminf(fminf(a.y, b.y), c.y), y_max = fmaxf(fmaxf(a.y, b.y), c.y);
  const float z_min = fminf(fminf(a.z, b.z), c.z), z_max = fmaxf(fmaxf(a.z, b.z), c.z);
  const float x_max = fmaxf(fmaxf(a.x, b.x), c.x);
  if (p.y < y_min || p.y > y_max || p.z < z_min || p.z > z_max || p.x > x_max) return false;
  const V3 e1 = vsub(b, a);
  const V3 e2 = vsub(c, a);
  // h = cross((1,0,0), e2)
  const V3 h = v3(fs(fm(0.0f, e2.z), fm(0.0f, e2.y)), fs(fm(0.0f, e2.x), fm(1.0f, e2.z)),
                  fs(fm(1.0f, e2.y), fm(0.0f, e2.x)));
  const float det = vdot(e1, h);
  if (fabsf(det) < 1.0e-12f) return false;
  const float inv_det = fd(1.0f, det);
  const V3 s = vsub(p, a);
  const float u = fm(inv_det, vdot(s, h));
  if (u < -1.0e-7f || u > 1.0f + 1.0e-7f) return false;
  const V3 q = v3(fs(fm(s.y, e1.z), fm(s.z, e1.y)), fs(fm(s.z, e1.x), fm(s.x, e1.z)),
                  fs(fm(s.x, e1.y), fm(s.y, e1.x)));
  const float v = fm(inv_det, vdot(v3(1.0f, 0.0f, 0.0f), q));
  if (v < -1.0e-7f || fa(u, v) > 1.0f + 1.0e-7f) return false;
  const float t = fm(inv_det, vdot(e2, q));
  return t > 1.0e-7f;
}

// Number of mesh triangles crossed by the +x ray from p (every node whose
// child box meets the ray {x >= p.x, y = p.y, z = p.z} is visited).
__device__ __forceinline__ int ray_x_crossings(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                               V3 p, int& overflow) {
  int stack[kTraversalStack];
  int sp = 0;
  int hits = 0;
  stack[sp++] = 0;
  while (sp > 0) {
    const int ref = stack[--sp];
    if (ref >= 0) {
      const float4* n = nodes + static_cast<size_t>(ref) * 8;
      const float4 hix = __ldg(n + 1), loy = __ldg(n + 2), hiy = __ldg(n + 3), loz = __ldg(n + 4),
                   hiz = __ldg(n + 5);
      const int4 ch = __ldg(reinterpret_cast<const int4*>(n + 6));
      const float hx[4] = {hix.x, hix.y, hix.z, hix.w}, ly[4] = {loy.x, loy.y, loy.z, loy.w},
                  hy[4] = {hiy.x, hiy.y, hiy.z, hiy.w}, lz[4] = {loz.x, loz.y, loz.z, loz.w},
                  hz[4] = {hiz.x, hiz.y, hiz.z, hiz.w};
      const int cr[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (cr[k] == kEmptyChild) continue;
        if (p.y < ly[k] || p.y > hy[k] || p.z < lz[k] || p.z > hz[k] || p.x > hx[k]) continue;
        if (sp < kTraversalStack) stack[sp++] = cr[k];
        else overflow = 1;
      }
    } else {
      const int first = leaf_first(ref), count = leaf_count(ref);
      const float4* t = tris + static_cast<size_t>(first) * 3;
      for (int i = 0; i < count; ++i) {
        const float4 a = __ldg(t + 3 * i), b = __ldg(t + 3 * i + 1), c = __ldg(t + 3 * i + 2);
        if (ray_x_hits(p, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z))) ++hits;
      }
    }
  }
  return hits;
}

}  // namespace dev
}  // namespace n2w

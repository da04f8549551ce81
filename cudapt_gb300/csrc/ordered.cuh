// The ordered walk: the reference's closest hit and any-hit answers, to the
// bit, from an eight-wide tree.
//
// Why it is exact.  TracePrimitive (trace.cuh) reaches leaves in one fixed
// order (right child first) and tests a leaf's triangles when the leaf's box
// and the boxes of all its ancestors pass IntersectAABB with the closest hit
// of that time.  Where boxes are nested, every slab distance of a child is
// rounded from a value inside its parent's, and rounding is monotone, so a
// leaf that passes its own test has passed all its ancestors' (the limit only
// shrinks): the leaf's own exact test alone decides.  Any other hierarchy over
// the same leaf order that never skips a passing leaf therefore gives the same
// sequence of triangle tests.  ordered_tree.cpp collapses the binary tree to
// eight children a node in that order, moves every child plane outwards past
// the rounding of both walks and stores it in 8 bits; leaf records hold the
// exact box, tested here with the reference's arithmetic.  Eight-wide nodes with
// 8-bit planes on a grid of their own, and the least-cost collapse, are Ylitie,
// Karras and Laine's ("Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs", HPG 2017); keeping the leaf order, and with it every
// answer, is not.
//
// What is left of the reference's limits: its 2048 pops.  A pop is the root or
// a child of an accepted inner node, and every accepted inner node lies in a
// visited wide node, so 1 + 2 * (inner nodes of the visited wide nodes) bounds
// the pops.  A walk whose bound passes 2048 (about 0.01 % of rays in the
// 332,180-triangle hall) is resolved by resolve_capped(), which counts the
// reference's pops exactly (kernels k_resolve and k_verify).  Scenes where that
// happens to more than a few per mille of random rays (walks_pass_bound), and
// scenes whose outward margin is large against their leaves (most_growth), keep
// the node-by-node walk.
//
// Cost: hall rays visit 22 wide nodes and 5-7 leaves on average where the
// binary walk pops 150-165 nodes one dependent fetch after another; a node
// is 96 bytes (three 32-byte loads) and a leaf 64.  What bounds it: issue slots
// (62 % used at 18 lanes per instruction in a hall bounce, 60 % of the integer
// and compare pipe) and the dependent fetches between them.  Eight children
// rather than four or six: 22, 28, 35 visits at about the same instructions per
// child, so the widest has the shortest chain.  Measured before -> after (whole
// calls): hall 1280x720 pass 4.72 -> 3.11 ms, interior 1024x768 4.49 -> 2.92,
// adaptive hall image 55.3 -> 37.1, unidirectional 333x217 image 9.37 -> 5.58,
// a million device rays in the hall 1.88 -> 1.18.
#pragma once
#include "gbpt_math.cuh"
#include "launch.h"
#include "ordered.h"
#include "trace.cuh"

namespace gbpt {

// Two float operations in one instruction (sm_100 and later), each lane
// rounded as the scalar operation.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b, float c) {
  const float2 r = __ffma2_rn(make_float2(a0, a1), make_float2(b, b), make_float2(c, c));
  d0 = r.x;
  d1 = r.y;
}

__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float d;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// byte k of w as the float 1 + byte * 2^-15 (one byte permute)
template <int k>
__device__ __forceinline__ float byte_float(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604 | (k << 4)));
}

constexpr uint32_t kPopCap = 2048;          // BVH_TRACE_MAX (include/cudaRTCommon.h:14)
constexpr uint32_t kPopStop = 4 * kPopCap;  // a bound this large ends a walk early, unresolved
// Longest direction component the node test takes (init_caller).  A plane step is cell /
// (|d| * limit), with cells of at least 2^-24 of the largest coordinate (itself
// at least 2^-10) and limits of at most 2^67: 2^-141 at this length.  The test's
// three roundings to subnormal numbers, 2^-150 each, stay below the 2^-7.4
// cells the planes' margin has left; from 2^92 on the products are zero.
constexpr float kOrdMaxDir = 0x1p40f;

// Walk state: the current group (child base and inner mask, leaf base and the
// mask of children still to visit, lowest bit first) in registers, groups with
// children left on the stack.
struct OrdWalk {
  gb::f3 o, d, inv;
  float minT;
  float scale;  // 1 / minT, held where the node test's products stay finite
  float bu, bv;
  uint32_t best;  // kNone: no hit
  uint32_t gA, gB, bound;
  int sp;
  static constexpr uint32_t kNone = 0xFFFFFFFFu;

  __device__ __forceinline__ void init(const DevScene& S, gb::f3 o_, gb::f3 d_, float maxDist) {
    using namespace gb;
    o = o_;
    d = d_;
    inv = mk(rcp_(escape_zero(d.x)), rcp_(escape_zero(d.y)), rcp_(escape_zero(d.z)));
    minT = maxDist;
    rescale(S);
    best = kNone;
    bu = bv = 0.f;
    sp = 0;
    bound = 1;
    // a group of one inner child: the root
    gA = 1u << 24;
    gB = 1u << 24;
    const float r = S.ordRange;
    // no finite direction at all: every slab distance is NaN and the reference's
    // root test fails
    if (isnan(inv.x) && isnan(inv.y) && isnan(inv.z)) gB = 0u;
    // an origin outside the range the planes' margin covers, or a NaN: unresolved
    else if (!(fabsf(o.x) <= r && fabsf(o.y) <= r && fabsf(o.z) <= r) || isnan(inv.x + inv.y + inv.z))
      gB = 0u, bound = kPopStop;
  }
  // A caller's ray: its direction may also be longer than the node test's products
  // carry.  The renderer's directions are quotients by their own length (or not
  // finite) and skip the test: 1 % of a hall pass.
  __device__ __forceinline__ void init_caller(const DevScene& S, gb::f3 o_, gb::f3 d_, float maxDist) {
    init(S, o_, d_, maxDist);
    if (fmax3_(fabsf(d.x), fabsf(d.y), fabsf(d.z)) > kOrdMaxDir) gB = 0u, bound = kPopStop;
  }

  // a limit above 1e20 lies beyond every plane (coordinates up to 1e9, slopes
  // up to 1e9), one below the range's 1e-7 keeps boxes it need not keep
  __device__ __forceinline__ void rescale(const DevScene& S) {
    scale = gb::rcp_(fmaxf(fminf(minT, 1e20f), S.ordRange * 1e-7f));
  }

  __device__ __forceinline__ bool hit() const { return best != kNone; }
  // the answer needs resolve_capped(): the reference may have run out of pops
  __device__ __forceinline__ bool capped() const { return bound > kPopCap; }
  __device__ __forceinline__ bool over() const { return (gB >> 24) == 0u && sp == 0; }
  // a resolved answer: the next step() reports the walk as over
  __device__ __forceinline__ void settle(bool hit, float4 h) {
    bound = 0;
    best = hit ? __float_as_uint(h.y) : kNone;
    minT = h.x;
    bu = h.z;
    bv = h.w;
  }

  __device__ __forceinline__ void pop(const uint2* stack) {
    if ((gB >> 24) == 0u && sp > 0) {
      const uint2 e = stack[--sp];
      gA = e.x;
      gB = e.y;
    }
  }

  // Tests the children of wide node `node` and makes the ones that may hold a
  // hit the current group.  Distances are scaled by `scale` = 1 / closest hit:
  // the third axis' saturating multiply-add then clips the interval to [0, 1]
  // for nothing, and a child is kept when its near distance is below its far
  // one (the margin of the planes makes that strict).  The kernel's scarce
  // pipe is the integer / compare one (byte permutes, selects, minima), so the
  // verdicts are taken as sign bits of packed subtractions and gathered by
  // three permutes per four children and one multiply for all eight.
  __device__ __forceinline__ void visit(const DevScene& S, uint32_t node) {
    using namespace gb;
    const float4* r = S.ord + 6 * (size_t)node;
    float4 A, B, X, Y;
    ldg_node(r, A, B);
    ldg_node(r + 2, X, Y);
    const float4 Z = __ldg(r + 4);
    const float ix = inv.x * scale, iy = inv.y * scale, iz = inv.z * scale;
    const float sx = A.w * ix, sy = B.x * iy, sz = B.y * iz;
    const float cx = fma_(A.x - o.x, ix, -sx), cy = fma_(A.y - o.y, iy, -sy), cz = fma_(A.z - o.z, iz, -sz);
    gA = __float_as_uint(B.z);
    const uint32_t leafWord = __float_as_uint(B.w);
    bound += 2u * (leafWord >> 24);
    const bool nx = __float_as_int(inv.x) < 0, ny = __float_as_int(inv.y) < 0, nz = __float_as_int(inv.z) < 0;
    uint32_t sign[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {  // children 0-3, 4-7
      const uint32_t lx = __float_as_uint(h ? X.y : X.x), hx = __float_as_uint(h ? X.w : X.z);
      const uint32_t ly = __float_as_uint(h ? Y.y : Y.x), hy = __float_as_uint(h ? Y.w : Y.z);
      const uint32_t lz = __float_as_uint(h ? Z.y : Z.x), hz = __float_as_uint(h ? Z.w : Z.z);
      const uint32_t ax = nx ? hx : lx, bx = nx ? lx : hx, ay = ny ? hy : ly, by = ny ? ly : hy, az = nz ? hz : lz,
                     bz = nz ? lz : hz;
      float n0x, n1x, n2x, n3x, n0y, n1y, n2y, n3y, f0x, f1x, f2x, f3x, f0y, f1y, f2y, f3y;
      fma2(n0x, n1x, byte_float<0>(ax), byte_float<1>(ax), sx, cx);
      fma2(n2x, n3x, byte_float<2>(ax), byte_float<3>(ax), sx, cx);
      fma2(n0y, n1y, byte_float<0>(ay), byte_float<1>(ay), sy, cy);
      fma2(n2y, n3y, byte_float<2>(ay), byte_float<3>(ay), sy, cy);
      fma2(f0x, f1x, byte_float<0>(bx), byte_float<1>(bx), sx, cx);
      fma2(f2x, f3x, byte_float<2>(bx), byte_float<3>(bx), sx, cx);
      fma2(f0y, f1y, byte_float<0>(by), byte_float<1>(by), sy, cy);
      fma2(f2y, f3y, byte_float<2>(by), byte_float<3>(by), sy, cy);
      const float n0 = fmax3_(n0x, n0y, fma_sat(byte_float<0>(az), sz, cz));
      const float n1 = fmax3_(n1x, n1y, fma_sat(byte_float<1>(az), sz, cz));
      const float n2 = fmax3_(n2x, n2y, fma_sat(byte_float<2>(az), sz, cz));
      const float n3 = fmax3_(n3x, n3y, fma_sat(byte_float<3>(az), sz, cz));
      const float f0 = fmin3_(f0x, f0y, fma_sat(byte_float<0>(bz), sz, cz));
      const float f1 = fmin3_(f1x, f1y, fma_sat(byte_float<1>(bz), sz, cz));
      const float f2 = fmin3_(f2x, f2y, fma_sat(byte_float<2>(bz), sz, cz));
      const float f3 = fmin3_(f3x, f3y, fma_sat(byte_float<3>(bz), sz, cz));
      const float2 d01 = __fadd2_rn(make_float2(n0, n1), make_float2(-f0, -f1));
      const float2 d23 = __fadd2_rn(make_float2(n2, n3), make_float2(-f2, -f3));
      // the four sign bytes in one word
      sign[h] = __byte_perm(__byte_perm(__float_as_uint(d01.x), __float_as_uint(d01.y), 0x0073),
                            __byte_perm(__float_as_uint(d23.x), __float_as_uint(d23.y), 0x0073), 0x5410);
    }
    // bits 3 and 7 of byte k: children k and 4 + k; the product moves them to
    // bits 24 + k and 28 + k (no two terms meet, so nothing carries)
    const uint32_t y = ((sign[0] >> 4) & 0x08080808u) | (sign[1] & 0x80808080u);
    gB = (leafWord & 0xFFFFFFu) | ((y * 0x00204081u) & 0xFF000000u);
  }

  // A leaf of the reference's walk: its exact box, then its triangles.  True
  // when one was accepted.
  __device__ __forceinline__ bool leaf(const DevScene& S, uint32_t rec) {
    using namespace gb;
    const float4* r = S.ordLeaf + 4 * (size_t)rec;
    float4 a, b, c, e;
    ldg_node(r, a, b);
    ldg_node(r + 2, c, e);
    const float t0x = (c.y - o.x) * inv.x, t1x = (e.x - o.x) * inv.x;
    const float t0y = (c.z - o.y) * inv.y, t1y = (e.y - o.y) * inv.y;
    const float t0z = (c.w - o.z) * inv.z, t1z = (e.z - o.z) * inv.z;
    float tb;
    if (!slab_hit(t0x, t1x, t0y, t1y, t0z, t1z, minT, tb)) return false;
    uint32_t id = __float_as_uint(e.w), left = 1;
    f3 P = mk(a.x, a.y, a.z), E0 = mk(a.w, b.x, b.y), E1 = mk(b.z, b.w, c.x);
    const bool many = (id & kOrdManyTris) != 0u;
    if (many) {
      id &= ~kOrdManyTris;
      left = __float_as_uint(a.x);
    }
    const f3 oe = o + eps * d;
    bool got = false;
    for (; left > 0; left--, id++) {
      if (many) {
        float4 p0, e0;
        ldg_node(S.tris + 4 * (size_t)id, p0, e0);
        const float4 e1 = __ldg(S.tris + 4 * (size_t)id + 2);
        P = mk(p0.x, p0.y, p0.z), E0 = mk(e0.x, e0.y, e0.z), E1 = mk(e1.x, e1.y, e1.z);
      }
      const f3 de2 = cross(d, E1);
      float div = dot(de2, E0);
      if (fabsf(div) < kLtEps9) continue;
      div = rcp_(div);
      const f3 t = oe - P;
      const f3 te1 = cross(t, E0);
      const float rT = dot(te1, E1) * div;
      if (!(rT >= 0.f && rT < minT)) continue;
      const float u = dot(de2, t) * div;
      if (u < 0.f || u > 1.f) continue;
      const float v = dot(te1, d) * div;
      if (v < 0.f || (u + v) > 1.f) continue;
      minT = rT;
      best = id;
      bu = u;
      bv = v;
      got = true;
      if (any) return true;
    }
    if (got) rescale(S);
    return got;
  }

  bool any;
  float eps;

  // The walk's next child is an inner node / a leaf (neither: it is over).
  __device__ __forceinline__ uint32_t next() const {
    const uint32_t m = gB >> 24;
    return m & (0u - m);
  }
  __device__ __forceinline__ bool wants_node() const { return (next() & (gA >> 24)) != 0u; }
  __device__ __forceinline__ bool wants_leaf() const { return (next() & ~(gA >> 24)) != 0u; }

  __device__ __forceinline__ void go_node(const DevScene& S, uint2* stack) {
    const uint32_t bit = next();
    const uint32_t node = (gA & 0xFFFFFFu) + __popc((gA >> 24) & (bit - 1u));
    gB ^= bit << 24;
    if (gB >> 24) stack[sp++] = make_uint2(gA, gB);
    visit(S, node);
  }

  // a walk far past the cap ends here: resolve_capped() answers
  __device__ __forceinline__ void stop_long() {
    if (bound >= kPopStop) {
      gB = 0u;
      sp = 0;
    }
  }

  __device__ __forceinline__ void go_leaf(const DevScene& S, uint2* stack) {
    const uint32_t bit = next();
    gB ^= bit << 24;
    const uint32_t rec = (gB & 0xFFFFFFu) + __popc(bit - 1u) - __popc((gA >> 24) & (bit - 1u));
    if (leaf(S, rec) && any) {
      gB = 0u;
      sp = 0;
    }
  }

  // One iteration of a lone thread; true when the walk is over.
  __device__ __forceinline__ bool step(const DevScene& S, uint2* stack) {
    pop(stack);
    if (wants_node()) go_node(S, stack);
    if (wants_leaf()) go_leaf(S, stack);
    stop_long();
    return over();
  }

  // One iteration of a warp's walks (`has`: this lane holds one): the lanes
  // whose next child is a node visit it, then the lanes whose next child is a
  // leaf test it, each part once and with the warp together.  True when this
  // lane's walk is over.  (Leaves held back until 8, 16 or 24 lanes have one:
  // hall frame 2.91 -> 2.96, 3.13, 3.65 ms.)
  __device__ __forceinline__ bool step_warp(const DevScene& S, uint2* stack, bool has) {
    if (has) {
      pop(stack);
      if (wants_node()) go_node(S, stack);
    }
    __syncwarp();
    if (has && wants_leaf()) go_leaf(S, stack);
    __syncwarp();
    return has && over();
  }
};

// The walks of up to four rays run by a warp, eight lanes a ray (group g = lanes
// 8g .. 8g + 7, all holding the same walk): lane c tests child c of the
// node and, of the leaves that come next in the order, the one in slot c; hits
// are then taken in the order.  The same tests on the same values as
// OrdWalk::visit and leaf.  A lone long walk is a chain of dependent fetches
// and instructions; this shortens the instructions' part (some 400 an iteration
// for a single lane) several times over.
__device__ __forceinline__ void coop_walk(const DevScene& S, OrdWalk& w, uint2* stack, bool live) {
  using namespace gb;
  const uint32_t lane = threadIdx.x & 31u, c = lane & 7u, group = lane & 24u;
  const bool nx = __float_as_int(w.inv.x) < 0, ny = __float_as_int(w.inv.y) < 0, nz = __float_as_int(w.inv.z) < 0;
  const uint32_t sel = 0x7604u | ((c & 3u) << 4);  // byte c & 3 as in byte_float
  const bool high = c >= 4u;
  for (;;) {
    w.stop_long();
    if (live) w.pop(stack);
    if (!__any_sync(0xffffffffu, live && !w.over())) break;
    const bool node = live && w.wants_node();
    bool hit = false;
    uint32_t nextA = w.gA, nextB = w.gB;
    if (node) {
      const uint32_t bit = w.next();
      const uint32_t id = (w.gA & 0xFFFFFFu) + __popc((w.gA >> 24) & (bit - 1u));
      const float4* r = S.ord + 6 * (size_t)id;
      float4 A, B, X, Y;
      ldg_node(r, A, B);
      ldg_node(r + 2, X, Y);
      const float4 Z = __ldg(r + 4);
      w.gB ^= bit << 24;
      if (w.gB >> 24) stack[w.sp++] = make_uint2(w.gA, w.gB);
      nextA = __float_as_uint(B.z);
      nextB = __float_as_uint(B.w);
      w.bound += 2u * (nextB >> 24);
      const float ix = w.inv.x * w.scale, iy = w.inv.y * w.scale, iz = w.inv.z * w.scale;
      const float sx = A.w * ix, sy = B.x * iy, sz = B.y * iz;
      const float cx = fma_(A.x - w.o.x, ix, -sx), cy = fma_(A.y - w.o.y, iy, -sy), cz = fma_(A.z - w.o.z, iz, -sz);
      auto plane = [&](float lo, float hi) {
        return __uint_as_float(__byte_perm(__float_as_uint(high ? hi : lo), 0x3F800000u, sel));
      };
      const float lx = plane(X.x, X.y), hx = plane(X.z, X.w), ly = plane(Y.x, Y.y), hy = plane(Y.z, Y.w),
                  lz = plane(Z.x, Z.y), hz = plane(Z.z, Z.w);
      const float n = fmax3_(fma_(nx ? hx : lx, sx, cx), fma_(ny ? hy : ly, sy, cy), fma_sat(nz ? hz : lz, sz, cz));
      const float f = fmin3_(fma_(nx ? lx : hx, sx, cx), fma_(ny ? ly : hy, sy, cy), fma_sat(nz ? lz : hz, sz, cz));
      hit = n < f;
    }
    const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> group) & 0xFFu;
    if (node) {
      w.gA = nextA;
      w.gB = (nextB & 0xFFFFFFu) | hits << 24;
      w.pop(stack);
    }
    // the leaves before the next inner child
    const uint32_t m = w.gB >> 24, im = w.gA >> 24, in = m & im;
    const uint32_t run = live ? m & ((in & (0u - in)) - 1u) & ~im : 0u;
    if (!__any_sync(0xffffffffu, run != 0u)) continue;
    bool cand = false;
    float near = 0.f, rT = 0.f, u = 0.f, v = 0.f;
    uint32_t id = 0;
    bool many = false;
    if ((run >> c) & 1u) {
      const float4* r = S.ordLeaf + 4 * (size_t)((w.gB & 0xFFFFFFu) + c - __popc(im & ((1u << c) - 1u)));
      float4 a, b, q, e;
      ldg_node(r, a, b);
      ldg_node(r + 2, q, e);
      id = __float_as_uint(e.w);
      many = (id & kOrdManyTris) != 0u;
      const bool box = slab_hit((q.y - w.o.x) * w.inv.x, (e.x - w.o.x) * w.inv.x, (q.z - w.o.y) * w.inv.y,
                                (e.y - w.o.y) * w.inv.y, (q.w - w.o.z) * w.inv.z, (e.z - w.o.z) * w.inv.z,
                                __uint_as_float(0x7f800000u), near);
      const f3 E0 = mk(a.w, b.x, b.y), E1 = mk(b.z, b.w, q.x), de2 = cross(w.d, E1);
      float div = dot(de2, E0);
      if (box && !many && !(fabsf(div) < kLtEps9)) {
        div = rcp_(div);
        const f3 t = (w.o + w.eps * w.d) - mk(a.x, a.y, a.z), te1 = cross(t, E0);
        rT = dot(te1, E1) * div;
        u = dot(de2, t) * div;
        v = dot(te1, w.d) * div;
        cand = rT >= 0.f && !(u < 0.f || u > 1.f) && !(v < 0.f || (u + v) > 1.f);
      }
    }
    const uint32_t manyRun = (__ballot_sync(0xffffffffu, many) >> group) & 0xFFu;
    if (manyRun) {  // leaves of several triangles: the run one leaf after another, by every lane of the group
      for (uint32_t left = run; left; left &= left - 1u)
        if (w.gB >> 24) w.go_leaf(S, stack);
      cand = false;
    }
    const bool took = run != 0u && !manyRun;
    if (took) w.gB ^= run << 24;
    for (uint32_t from = 0;;) {
      const uint32_t ok = __ballot_sync(0xffffffffu, cand && c >= from && near < w.minT && rT < w.minT);
      if (ok == 0u) break;
      const uint32_t mine = (ok >> group) & 0xFFu;
      const int src = mine ? (int)group + __ffs((int)mine) - 1 : (int)lane;
      const float t1 = __shfl_sync(0xffffffffu, rT, src), u1 = __shfl_sync(0xffffffffu, u, src),
                  v1 = __shfl_sync(0xffffffffu, v, src);
      const uint32_t id1 = __shfl_sync(0xffffffffu, id, src);
      if (mine) {
        w.minT = t1;
        w.bu = u1;
        w.bv = v1;
        w.best = id1;
        w.rescale(S);
        from = ((uint32_t)src & 7u) + 1u;
        if (w.any) {
          w.gB = 0u;
          w.sp = 0;
          cand = false;
          from = 8u;
        }
      }
    }
  }
}

// The walks of a warp's last few lanes (at most four bits of `live`) to their
// ends, eight lanes each: the k-th live lane's walk and stack are copied to
// lanes 8k .. 8k + 7 and its result is taken back.  Warp-uniform call.
__device__ __forceinline__ void gather_walks(const DevScene& S, OrdWalk& w, uint2* stack, uint32_t live) {
  using namespace gb;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t m = live;
  for (uint32_t k = lane >> 3; k > 0; k--) m &= m - 1u;
  const bool have = m != 0u;
  const int src = have ? __ffs((int)m) - 1 : (int)lane;
  const auto from = [src](float x) { return __shfl_sync(0xffffffffu, x, src); };
  const auto fromU = [src](uint32_t x) { return __shfl_sync(0xffffffffu, x, src); };
  const int mine = (live >> lane) & 1u ? w.sp : 0;
  const int deepest = __reduce_max_sync(0xffffffffu, mine);
  // entry i moves to entry i, read before it is written: no second stack
  for (int i = 0; i < deepest; i++) {
    const uint2 e = i < mine ? stack[i] : make_uint2(0u, 0u);
    stack[i] = make_uint2(fromU(e.x), fromU(e.y));
  }
  w.o = mk(from(w.o.x), from(w.o.y), from(w.o.z));
  w.d = mk(from(w.d.x), from(w.d.y), from(w.d.z));
  w.inv = mk(from(w.inv.x), from(w.inv.y), from(w.inv.z));
  w.minT = from(w.minT);
  w.scale = from(w.scale);
  w.bu = from(w.bu);
  w.bv = from(w.bv);
  w.best = fromU(w.best);
  w.gA = fromU(w.gA);
  w.gB = fromU(w.gB);
  w.bound = fromU(w.bound);
  w.sp = __shfl_sync(0xffffffffu, mine, src);
  w.any = __shfl_sync(0xffffffffu, (int)w.any, src) != 0;
  w.eps = from(w.eps);
  coop_walk(S, w, stack, have);
  // the ray goes back too: a walk past the pop bound is run again from it
  const int home = (int)(8u * (uint32_t)__popc(live & ((1u << lane) - 1u))) & 31;
  const auto back = [home](float x) { return __shfl_sync(0xffffffffu, x, home); };
  w.o = mk(back(w.o.x), back(w.o.y), back(w.o.z));
  w.d = mk(back(w.d.x), back(w.d.y), back(w.d.z));
  w.minT = back(w.minT);
  w.bu = back(w.bu);
  w.bv = back(w.bv);
  w.best = __shfl_sync(0xffffffffu, w.best, home);
  w.bound = __shfl_sync(0xffffffffu, w.bound, home);
  w.any = __shfl_sync(0xffffffffu, (int)w.any, home) != 0;
  w.eps = back(w.eps);
  w.gB = 0u;
  w.sp = 0;
}

// The reference's answer for a ray whose walk may have run out of pops, by a
// block.  The binary tree is searched level by level without the closest hit
// (its limit only ever rejects more): the accepted inner nodes are kept with
// their entry distances, the triangles hit with their leaves.  In the
// reference's order (leaves right to left, nodes are numbered left to right)
// those hits give the sequence of closest-hit changes, the k-th at leaf at_k;
// an inner node whose subtree ends before node E was accepted when its entry
// lay below the limit left by the changes with at_k >= E, and a node is
// popped before or at leaf at_k exactly when its own E > at_k.  With at most
// 2048 pops the last change stands, otherwise the last one whose leaf was
// among the first 2048, found by halving.  About 25 dependent rounds (the
// tree's depth) in place of up to 2048: 20 us of search and 8 of ordering and
// counting for a hall ray of 540-1410 accepted nodes and 30-70 hits, the lists
// sized so that four blocks share an SM.  A search that overflows them takes
// the reference's walk instead.
constexpr uint32_t kCapThreads = 256, kCapFront = 1024, kCapNodes = 2048, kCapHits = 192;
struct CapShared {
  uint2 front[2][kCapFront];  // {node, end of its subtree}
  float near[kCapNodes];
  uint32_t end[kCapNodes], mid[kCapNodes];  // end of the subtree, its right child
  float4 hit[kCapHits];                     // t, triangle, u, v
  float hitNear[kCapHits], dist[kCapHits];
  uint32_t hitLeaf[kCapHits], order[kCapHits], at[kCapHits], what[kCapHits];
  uint32_t frontN[3], nodeN, hitN, over, changes, sum[32];
  float4 answer;
  uint32_t found;
};

__device__ __forceinline__ uint32_t cap_sum(CapShared& c, uint32_t v) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31u) == 0u) c.sum[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  for (uint32_t k = 0; k < blockDim.x / 32; k++) t += c.sum[k];
  return t;
}

// every thread of the block, with the same arguments; the answer is in
// c.found / c.answer afterwards
__device__ __forceinline__ void resolve_capped(const DevScene& S, CapShared& c, gb::f3 o, gb::f3 d, float maxDist,
                                               float eps, bool any) {
  using namespace gb;
  const uint32_t tid = threadIdx.x, stride = blockDim.x;
  const f3 inv = mk(rcp_(escape_zero(d.x)), rcp_(escape_zero(d.y)), rcp_(escape_zero(d.z)));
  const f3 oe = o + eps * d;
  __syncthreads();
  if (tid == 0) {
    c.front[0][0] = make_uint2(0u, S.nodeN);
    c.frontN[0] = 1u;
    c.frontN[1] = c.frontN[2] = c.nodeN = c.hitN = c.over = c.found = c.changes = 0u;
  }
  __syncthreads();
  // level L: frontier L & 1, its size in counter L % 3, the next level's in
  // (L + 1) % 3; the third is zeroed meanwhile, so a level needs one barrier
  uint32_t level = 0;
  for (;; level++) {
    const int cur = (int)(level & 1u);
    const uint32_t n = min(c.frontN[level % 3u], kCapFront);
    if (n == 0u) break;  // (an overflow ends by itself: nothing more is pushed)
    uint32_t* nextN = &c.frontN[(level + 1u) % 3u];
    if (tid == 0) c.frontN[(level + 2u) % 3u] = 0u;
    for (uint32_t i = tid; i < n; i += stride) {
      const uint2 e = c.front[cur][i];
      const uint32_t id = e.x, E = e.y;
      float4 a, b;
      ldg_node(S.nodes + 2 * (size_t)id, a, b);
      float tb;
      if (!slab_hit((a.x - o.x) * inv.x, (b.x - o.x) * inv.x, (a.y - o.y) * inv.y, (b.y - o.y) * inv.y,
                    (a.z - o.z) * inv.z, (b.z - o.z) * inv.z, maxDist, tb))
        continue;
      const uint32_t off = __float_as_uint(a.w), tn = __float_as_uint(b.w);
      if (tn == 0u) {
        if (*(volatile uint32_t*)&c.over) continue;
        const uint32_t k = atomicAdd(&c.nodeN, 1u);
        const uint32_t f = k < kCapNodes ? atomicAdd(nextN, 2u) : kCapFront;
        if (f + 2u > kCapFront) {
          c.over = 1u;
          continue;
        }
        c.near[k] = tb;
        c.end[k] = E;
        c.mid[k] = id + off;
        // the tree is cold here (the walks use their own): fetch ahead
        asm volatile("prefetch.global.L2 [%0];" ::"l"(S.nodes + 2 * (size_t)(id + 1u)));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(S.nodes + 2 * (size_t)(id + off)));
        c.front[cur ^ 1][f] = make_uint2(id + 1u, id + off);
        c.front[cur ^ 1][f + 1u] = make_uint2(id + off, E);
        continue;
      }
      for (uint32_t t = off; t < off + tn; t++) {
        float4 p0, e0;
        ldg_node(S.tris + 4 * (size_t)t, p0, e0);
        const float4 e1 = __ldg(S.tris + 4 * (size_t)t + 2);
        const f3 E0 = mk(e0.x, e0.y, e0.z), E1 = mk(e1.x, e1.y, e1.z), de2 = cross(d, E1);
        float div = dot(de2, E0);
        if (fabsf(div) < kLtEps9) continue;
        div = rcp_(div);
        const f3 q = oe - mk(p0.x, p0.y, p0.z), te1 = cross(q, E0);
        const float rT = dot(te1, E1) * div;
        if (!(rT >= 0.f && rT < maxDist)) continue;
        const float u = dot(de2, q) * div;
        if (u < 0.f || u > 1.f) continue;
        const float v = dot(te1, d) * div;
        if (v < 0.f || (u + v) > 1.f) continue;
        const uint32_t k = atomicAdd(&c.hitN, 1u);
        if (k >= kCapHits) {
          c.over = 1u;
          continue;
        }
        c.hit[k] = make_float4(rT, __uint_as_float(t), u, v);
        c.hitNear[k] = tb;
        c.hitLeaf[k] = id;
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (c.over != 0u) {
    if (tid == 0) {
      TraceHit h;
      uint32_t nn = 0, nt = 0;
      const bool hit = any ? trace_ref<true, false>(S, o, d, maxDist, eps, false, h, nn, nt)
                           : trace_ref<false, false>(S, o, d, maxDist, eps, false, h, nn, nt);
      c.found = hit ? 1u : 0u;
      if (hit) c.answer = make_float4(h.t, __uint_as_float(h.tri), h.u, h.v);
    }
    __syncthreads();
    return;
  }
  // the hits in the reference's order: leaves from the largest node id down,
  // inside a leaf by triangle
  const uint32_t nh = c.hitN;
  for (uint32_t i = tid; i < nh; i += stride) {
    const uint32_t leaf = c.hitLeaf[i], t = __float_as_uint(c.hit[i].y);
    uint32_t rank = 0;
    for (uint32_t j = 0; j < nh; j++)
      rank += c.hitLeaf[j] > leaf || (c.hitLeaf[j] == leaf && __float_as_uint(c.hit[j].y) < t) ? 1u : 0u;
    c.order[rank] = i;
  }
  __syncthreads();
  // the changes, by one warp: of the hits in order the first that is closer,
  // in a leaf whose box passes (or whose triangles are being tested already)
  if (tid < 32u) {
    float minT = maxDist;
    uint32_t open = 0xFFFFFFFFu, n = 0;
    for (uint32_t base = 0; base < nh; base += 32u) {
      const bool in = base + tid < nh;
      const uint32_t i = in ? c.order[base + tid] : 0u;
      const float t = in ? c.hit[i].x : 0.f, box = in ? c.hitNear[i] : 0.f;
      const uint32_t leaf = in ? c.hitLeaf[i] : 0u;
      uint32_t from = 0;
      for (;;) {
        const bool ok = in && tid >= from && t < minT && (leaf == open || box < minT);
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        if (m == 0u) break;
        const int src = __ffs((int)m) - 1;
        minT = __shfl_sync(0xffffffffu, t, src);
        open = __shfl_sync(0xffffffffu, leaf, src);
        from = (uint32_t)src + 1u;
        if (tid == (uint32_t)src) {
          c.dist[n] = t;
          c.at[n] = leaf;
          c.what[n] = i;
        }
        n++;
        if (any) break;
      }
      if (any && n) break;
    }
    if (tid == 0) c.changes = n;
  }
  __syncthreads();
  const uint32_t n = c.changes;
  if (n == 0u) return;
  // pops of nodes whose subtree ends after `upto`
  auto pops = [&](uint32_t upto) {
    uint32_t v = tid == 0 ? 1u : 0u;  // the root
    for (uint32_t i = tid; i < c.nodeN; i += stride) {
      const uint32_t E = c.end[i];
      uint32_t lo = 0, hi = any ? 0u : n;  // changes with at >= E
      while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        if (c.at[m] >= E)
          lo = m + 1u;
        else
          hi = m;
      }
      if (lo > 0u && !(c.near[i] < c.dist[lo - 1u])) continue;
      v += (E > upto ? 1u : 0u) + (c.mid[i] > upto ? 1u : 0u);
    }
    return cap_sum(c, v);
  };
  uint32_t keep = n;  // changes that count
  if (pops(0u) > kPopCap) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
      const uint32_t m = (lo + hi + 1u) >> 1;
      if (pops(c.at[m - 1u]) <= kPopCap)
        lo = m;
      else
        hi = m - 1u;
    }
    keep = lo;
  }
  if (tid == 0 && keep > 0u) {
    c.found = 1u;
    c.answer = c.hit[c.what[keep - 1u]];
  }
  __syncthreads();
}

// Closest hit of one ray by one thread; `open` (when given) is set and nothing
// answered for a walk past the bound, which otherwise takes the reference's walk.
__device__ __forceinline__ bool trace_ord(const DevScene& S, gb::f3 o, gb::f3 d, float maxDist, float eps,
                                          TraceHit& h, bool* open = nullptr) {
  OrdWalk w;
  uint2 stack[kOrdStack];
  w.any = false;
  w.eps = eps;
  w.init_caller(S, o, d, maxDist);
  while (!w.step(S, stack)) {
  }
  if (w.capped()) {
    if (open) {
      *open = true;
      return false;
    }
    uint32_t nn = 0, nt = 0;
    return trace_ref<false, false>(S, o, d, maxDist, eps, false, h, nn, nt);
  }
  if (!w.hit()) return false;
  h.t = w.minT;
  h.tri = w.best;
  h.w = 1.f - w.bu - w.bv;
  h.u = w.bu;
  h.v = w.bv;
  return true;
}

// Walk kinds of the wavefront kernels: the reference's order node by node
// (counters on, or a scene or camera the ordered walk does not take), the
// opt-in wide order, and the ordered walk.  Walk type, stack entry type and
// stack depth of each.
enum : int { kWalkRef = 0, kWalkWide = 1, kWalkOrd = 2 };
template <int kKind>
struct WalkOf {
  using type = Walk;
  using Entry = uint32_t;
  static constexpr int kDepth = 32;
};
template <>
struct WalkOf<kWalkWide> {
  using type = Walk4;
  using Entry = uint2;
  static constexpr int kDepth = (int)kWideDepth;
};
template <>
struct WalkOf<kWalkOrd> {
  using type = OrdWalk;
  using Entry = uint2;
  static constexpr int kDepth = (int)kOrdStack;
};

// A walk of any kind started and stepped alike.
template <int kKind>
__device__ __forceinline__ void start_walk(const DevScene& S, typename WalkOf<kKind>::type& w, gb::f3 o, gb::f3 d,
                                           float maxDist, bool any, typename WalkOf<kKind>::Entry* stack) {
  if constexpr (kKind == kWalkOrd) {
    w.any = any;
    w.eps = gb::kBias;
    w.init(S, o, d, maxDist);
  } else {
    w.init(o, d, maxDist, gb::kBias, stack);
  }
}
template <int kKind, bool kCount>
__device__ __forceinline__ bool step_walk(const DevScene& S, typename WalkOf<kKind>::type& w,
                                          typename WalkOf<kKind>::Entry* stack, bool any, uint32_t& nodes,
                                          uint32_t& tris) {
  if constexpr (kKind == kWalkOrd)
    return w.step(S, stack) && !w.capped();
  else
    return w.template step<kCount>(S, stack, any, nodes, tris);
}

}  // namespace gbpt

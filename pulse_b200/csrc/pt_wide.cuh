// pt_wide.cuh -- closest-hit and occlusion traversal over eight-wide nodes.
//
// The trees of the scene stay the reference's binary ones (same leaves, same
// node arrays); wide.cu collapses each into nodes of up to eight children with
// their boxes quantized to 8 bits per plane, rounded outwards (96 bytes against
// the 448 of the seven binary interior nodes it stands for).  A ray visits
// about a third of the nodes, each with one set of independent loads.  (Wide nodes with
// quantized boxes on a power-of-two grid: Ylitie, Karras and Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs", 2017.)
//
// The result is the reference's bit for bit although nodes are visited in
// another order.  Within one BLAS (o, d object space, t local; the TLAS level
// below is the same argument with instances for triangles):
//   * The reference tests a triangle only in leaves whose ancestor boxes all
//     pass its slab test and were entered before the record t fell to the
//     box's t_min.  Boxes nest, and IEEE subtraction and division are
//     monotone, so the leaf's own box has the largest t_min and the smallest
//     t_max of its chain: a leaf box that passes (t_max >= t_min, t_max > 0)
//     vouches for its ancestors.
//   * Let A be the nearest hit, m its leaf box's t_min, M = max(t_A, m).  If the box
//     passes, the reference can only end with another hit B if B kept it out of A's
//     leaf or came first with the same t: t_A <= t_B <= M.  Hits up to a gate a little
//     beyond the nearest one (wide_gate) are looked at, and a second one in that interval
//     makes the ray ambiguous, unless both lie in one leaf: then the nearer one is the reference's.
//   * The traversal finds candidates: triangles whose test may pass (exact up to its
//     division, then with a margin), with t and the world distance to a few roundings,
//     which the gates cover.  When the ray ends its candidate is verified
//     (wide_verify): the reference's arithmetic accepts the triangle, its leaf boxes pass
//     and their t_min are within the gates.  Only the candidate of the ray's
//     nearest instance needs it: one of another instance that fails can only give way to
//     a farther hit.  Ambiguous rays and those that fail are traced again by the
//     binary traversal (1 in 100,000 of the 1080p sphere frame).
//   * Every leaf holding a hit with t <= M must be visited.  Quantized boxes
//     contain the exact ones with 1/64 of a quantum to spare, the far planes are
//     scaled by 1 + 2e-6 (the rounding of a plane's t is below 5e-7 of it
//     plus 1/100 of a quantum), and boxes are skipped only beyond the gate and a slack:
//     the computed t of a hit may lie before its box by the rounding of the reference's
//     triangle test, which for a ray along the plane of a large triangle is a good part of
//     the distance.  triangle_slack (wide.cu) bounds it by (t + longer edge) * slack; meshes
//     whose triangles have no such bound are not culled by distance at all.  (A slack of at most
//     0.02 answered 1 in 10,000 rays along triangles of 20 to 200 units wrongly.  Without it
//     720p frames of a terrain of 400 units in 8 to 96 squares a side take 0 to 5% longer
//     than with it, 16% at worst; the binary trees take 1.2 to 1.6 times as long.  Scenes
//     of many such triangles keep the binary trees: decide_wide, api.cu.)  Left out is a hit
//     whose ray passes beside the triangle by a rounding and enters its box later by that
//     over the direction's component, if that is below 0.01.
// Rays and scenes outside these arguments (a direction that is not
// normalized, coordinates above 1e9, boxes that do not nest, transforms that are
// not affine or nearly singular, stacks or iteration caps that bind) take the binary
// traversal: per ray here, per launch in the host's choice of kernel.
#pragma once
#include "pt_trace.cuh"

namespace pt {

// Node words (24, 96 bytes):
//   0-2 origin, 3 exponents of the quanta (biased, + 15; 3 bytes) | interior children << 24 | leaf children << 28,
//   4 first interior child | axis << 22 (they are consecutive, sorted along the axis), 8-19 the planes
//   qlo.x[8] qhi.x[8] qlo.y[8] qhi.y[8] qlo.z[8] qhi.z[8].
// Interior children take the slots from 0 up, leaves those from 7 down; leaf r = 7 - slot
// has its reference in word 5, 6, 7, 20, 21, 22, 23 or 4: triangle count << 26 | first triangle
// slot in a BLAS, the instance in the TLAS (bit 31: of a mesh with more than the least
// slack).  Node indexes and triangle slots are those of the
// scene's concatenated arrays (relocate, wide.cu).
constexpr uint32_t kWideFirstBits = 26, kWideMaxCount = 63;
constexpr uint32_t kWideFirstMask = (1u << kWideFirstBits) - 1u;
constexpr uint32_t kWideRootLeaf = 0xffffffffu;  // leaf index of a tree that is one leaf: no box was tested
constexpr uint32_t kWideNodeWords = 24;
__host__ __device__ constexpr uint32_t wide_ref_word(uint32_t r) { return r < 3u ? 5u + r : r < 7u ? 17u + r : 4u; }

// Within a BLAS, a group of children still to be visited is one stack word: an interior
// group is the first interior child's index, the axis they are sorted along and a hit
// bit per slot; a leaf group (never on the stack) is the node's own index, axis 3 and the
// hit bits.  Indexes take 22 bits.
constexpr uint32_t kWideIndexBits = 22;
constexpr uint32_t kWideIndexMask = (1u << kWideIndexBits) - 1u;

// In the TLAS, whose boxes overlap and whose leaves are costly, every child hit is a
// stack word of its own, the nearest on top: the entry distance's upper 14
// bits (rounded down: entries beyond the record are dropped when popped), then
// interior: child index << 1; leaf: instance << 1 | 1.  The distance of a child that
// holds an instance of more than the least slack is lowered by the largest slack of the scene.
// Where the children hit do not fit, one is gone on with and the node itself is the
// entry of the rest, to be visited again without the children that were missed or are done:
// kTopAgain | those << 17 | node (distances stay below 2^97, boxes lying within 1e9, so no
// entry's upper three bits are all ones).  That takes one entry a level at most, beyond
// the cfg.stack_top entries up to which children are pushed.
constexpr uint32_t kTopIndexBits = 17, kTopIndexMask = (1u << kTopIndexBits) - 1u;
constexpr uint32_t kTopAgain = 0xe0000000u;
constexpr uint32_t kLooseRef = 0x80000000u;
constexpr float kLeastSlack = 1e-4f;
// Node word 4 of the TLAS from this bit: the interior children that hold a loose instance.
constexpr uint32_t kTopLooseShift = 24;
// A slack that culls nothing (boxes lie within 4e9 of a ray's origin), and up to which one bounds
// a hit (wide.cu).
constexpr float kNoSlackBound = 1e15f, kMostSlack = 0.5f;
// Entries up to which children are pushed: 16 for trees of up to 3 levels (the 1080p
// sphere frame: 9.3 ms, with 24 and the less L1 they leave 9.45), 24 for deeper ones as far as
// the stack of both levels stays within 36 words, the most with which four blocks fit an SM
// (the 4K terrain frame 23.9 ms, with 38 words 26.8), and 12 at least.  640 x 360 frames of
// 4,000 / 30,000 / 100,000 instances with 24: 4.1 / 6.9 / 11.7 ms; 12: 4.0 / 7.3 / 14.1
// (the binary traversal 6.7 / 12.0 / 23.7).  Before kTopAgain, rays that overflowed were
// traced again by the binary traversal: 4.1 / 14.3 / 39.7 ms.
constexpr uint32_t kWideStack = 36, kTopLeast = 12, kTopShallow = 16, kTopMost = 24;

// ------------------------------------------------------------- ray pools
// A warp keeps kPool rays in shared memory (word k of slot s at [k * kPool + s]), two
// for each lane, and performs one action per step for up to 32 of those that wait
// for it: with four classes of actions (node, triangles, instance, other) the
// fullest one mostly fills the warp: 22 slots a step and 18 threads an instruction in the
// first launches of the sphere frame, where one ray per lane in registers left 13 to
// 14.  Three rays a lane took 9.74 ms against 9.32 with two.
constexpr uint32_t kPool = 64;

// An instance's record for entering it (DevScene::inst_wide), 96 bytes: its
// world-to-object matrix (affine: the first three columns' w hold the mesh's slack in units of
// its space and the margins e1, e0 of its distances, 0 unless it is sheared), (root group of the
// mesh's tree, or 0 and its only leaf's reference, slack of the mesh, mesh id), (first triangle
// slot, first binary node, TLAS leaf node or kWideRootLeaf, scene_prep.cuh's wide_leaves).
constexpr uint32_t kWideInstRows = 6;

enum WideWord : uint32_t {
  kwOX, kwOY, kwOZ, kwDX, kwDY, kwDZ,  // ray of the level
  kwCull,                              // box entry bound of the level
  kwGrp,                               // current group
  kwCur,                               // current leaf: elements left << 26 | next element; TLAS: node (children
                                       // not to visit << 17) or instance
  kwSp,                                // stack entries | those of the TLAS level << 7 | instance << 14 | in a BLAS << 31
  kwLen, kwSlack,                      // object distance per world distance; slack of the mesh
  kwLimit,                             // of an occlusion query, else 3e38
  kwFar,                               // box entry bound of an occlusion query (world), else infinity
  kwEps,                               // rounding of world distances
  kwRecT, kwRecSlot, kwRecInst,        // nearest candidate: world distance, triangle slot, instance | scene << 20
  kwId,                                // the kernel's
  kWideWords,
  kwU = kwOX, kwV = kwOY               // of a verified hit
};
constexpr uint32_t kInstBits = 17, kInstMask = (1u << kInstBits) - 1u;
// Action classes of a slot.  kwShade: the kernel's own step.
enum WideAct : uint32_t {
  kwNode = 0, kwTriangles = 1, kwInstance = 2, kwVerify = 3, kwRedo = 4, kwShade = 5, kwEmpty = 6, kwDone = 7
};

// Words of a warp's pool: the rays with their stacks, the slots' classes and the step's list.
__host__ __device__ constexpr uint32_t wide_pool_words(uint32_t stack) {
  return (kWideWords + stack) * kPool + kPool / 4 + 32 / 4;
}

struct WideRay {
  uint32_t* p;  // the slot's first word
  __device__ __forceinline__ uint32_t u(uint32_t k) const { return p[k * kPool]; }
  __device__ __forceinline__ float f(uint32_t k) const { return __uint_as_float(u(k)); }
  __device__ __forceinline__ float3 f3(uint32_t k) const { return v3(f(k), f(k + 1), f(k + 2)); }
  __device__ __forceinline__ void set(uint32_t k, uint32_t v) const { p[k * kPool] = v; }
  __device__ __forceinline__ void setf(uint32_t k, float v) const { set(k, __float_as_uint(v)); }
  __device__ __forceinline__ void setf3(uint32_t k, float3 v) const { setf(k, v.x); setf(k + 1, v.y); setf(k + 2, v.z); }
  __device__ __forceinline__ uint32_t& stack(uint32_t i) const { return p[(kWideWords + i) * kPool]; }
};

struct Words8 { uint32_t w[8]; };
__device__ __forceinline__ Words8 ldg256(const uint4* p) {
  Words8 r;
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
      : "l"(p));
  return r;
}

// 1 / x for box tests; a zero or tiny component gets a large reciprocal of its
// sign (its slab then spans the ray wherever the exact one does).
__device__ __forceinline__ float wide_rcp(float x) {
  const float a = fabsf(x) < 1e-18f ? copysignf(1e-18f, x) : x;
  return __fdividef(1.0f, a);
}

__device__ __forceinline__ bool wide_ray_ok(float3 o, float3 d) {
  const float dd = dot(d, d);
  return fabsf(dd - 1.0f) < 1e-4f && max_abs3(o) <= 1e9f && o.x == o.x && o.y == o.y && o.z == o.z;
}

// Whether the reference's slab test without its record comparison (src/utilities.wgsl:405-426)
// passes a box and its t_min is at most bound.  Answered from planes by reciprocals, within
// 4e-7 of the reference's quotients, where every comparison holds by 2e-6 (the planes of one
// axis need none: their quotients are ordered like them, so boxes without thickness are
// answered too); rays that pass an edge closer, or fail, take the exact test.
__device__ __forceinline__ bool enters_box(float3 o, float3 d, const float4* node, float bound) {
  const float4 lo = __ldg(node), hi = __ldg(node + 1);
  const float3 r = v3(__fdividef(1.0f, d.x), __fdividef(1.0f, d.y), __fdividef(1.0f, d.z));
  const float ax = (lo.x - o.x) * r.x, bx = (hi.x - o.x) * r.x;
  const float ay = (lo.y - o.y) * r.y, by = (hi.y - o.y) * r.y;
  const float az = (lo.z - o.z) * r.z, bz = (hi.z - o.z) * r.z;
  const float nx = fminf(ax, bx), ny = fminf(ay, by), nz = fminf(az, bz);
  const float fx = fmaxf(ax, bx), fy = fmaxf(ay, by), fz = fmaxf(az, bz);
  const float tn = fmaxf(fmaxf(nx, ny), nz), tf = fminf(fminf(fx, fy), fz);
  const float most = fmaxf(fmaxf(fabsf(ax), fabsf(bx)),
                           fmaxf(fmaxf(fabsf(ay), fabsf(by)), fmaxf(fabsf(az), fabsf(bz))));
  const float gap = fminf(fminf(fx - fmaxf(ny, nz), fy - fmaxf(nx, nz)), fz - fmaxf(nx, ny));
  const float least = fminf(fminf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
  if (gap > 2e-6f * most && tf > 1e-30f && tn + 2e-6f * fabsf(tn) <= bound && most < 1e28f && least > 1e-18f) return true;
  const float t = ray_aabb(o, d, 1e30f, lo, hi);
  return t < 1e30f && t <= bound;
}

constexpr uint32_t kInBlas = 1u << 31;

// The end of the interval from a nearest hit at world distance t in which another one
// makes the ray ambiguous: beyond the rounding of distances and of boxes' t_min.  eps (kwEps) is
// 1e-6 of the largest world coordinate, and 1.6e-6 of the largest object coordinate in world
// units, of the ray's origin in the instances entered so far: distances pass through their
// transforms.  A sheared instance multiplies the roundings and has a margin of its own (e1 and e0 of
// its record; without it, of rays onto two sheared instances that coincide 1 in 500 to
// 30,000 took the wrong one for axes of 1 to 0.001 or 0.01).
__device__ __forceinline__ float wide_gate(float t, float eps) { return t * 1.0000025f + eps; }

// The bound of boxes whose hits may be found up to the slack before them.
__device__ __forceinline__ float wide_bound(float t, float slack) { return t * (1.0f + slack) + slack; }

// Whether a hit at world distance t decides an occlusion query, before its exact distance
// is known: it lies before the limit by world_cull's margins.  Never for other queries (their
// bound is infinite and the difference no number).
__device__ __forceinline__ bool wide_decides(const WideRay& R, float t) {
  return t < 2.0f * R.f(kwLimit) - R.f(kwFar);
}

// The level becomes the TLAS.
__device__ __forceinline__ void wide_world(const WideRay& R, const DevScene& S, float3 wo, float3 wd, float rec_t,
                                           float far) {
  R.setf3(kwOX, wo);
  R.setf3(kwDX, wd);
  R.setf(kwCull, fminf(wide_bound(rec_t, S.wide_slack), far));
}

// Begin a ray of a scene in a slot; its first class.  limit < 1e29 makes it an occlusion
// query.
__device__ __forceinline__ uint32_t wide_begin(const WideRay& R, uint32_t scene, const DevScene& S, float3 wo,
                                               float3 wd, float limit) {
  const float far = limit < 1e29f ? world_cull(limit, wo) : __int_as_float(0x7f800000);
  wide_world(R, S, wo, wd, 1e30f, far);
  R.set(kwSp, 0u);
  R.setf(kwRecT, 1e30f);
  R.set(kwRecInst, scene << 20);
  R.set(kwCur, 0u);  // the root node
  R.setf(kwFar, far);
  R.setf(kwEps, 1e-6f * max_abs3(wo));
  R.setf(kwLimit, limit < 1e29f ? limit : 3.0e38f);
  if (!(limit > 0.0f)) return kwDone;
  return wide_ray_ok(wo, wd) ? kwNode : kwRedo;
}

// The next leaf of a leaf group whose hit bits are not all zero, taken out of the group.
__device__ __forceinline__ uint32_t wide_leaf(const DevScene& S, uint32_t& grp) {
  const uint32_t r = __clz(grp);  // 7 - slot of the highest hit bit
  grp &= ~(0x80000000u >> r);
  const uint32_t* w =
      reinterpret_cast<const uint32_t*>(S.wide_blas + (size_t)(grp & kWideIndexMask) * (kWideNodeWords / 4));
  return __ldg(w + wide_ref_word(r));
}

// The next group of the BLAS, or its end; kwSp holds the new stack.
__device__ __forceinline__ uint32_t wide_pop(const WideRay& R, uint32_t spx) {
  const bool some = (spx & 0x7fu) > ((spx >> 7) & 0x7fu);
  if (some) {
    --spx;
    R.set(kwGrp, R.stack(spx & 0x7fu));
  }
  R.set(kwSp, spx);
  return some ? kwNode : kwInstance;
}

// The next entry of the TLAS stack that is not beyond the bound, or the ray's end.
__device__ __forceinline__ uint32_t wide_top_pop(const WideRay& R, uint32_t sp, float bound, float rec_t) {
  uint32_t next = kwDone;
  while (sp > 0u) {
    const uint32_t e = R.stack(--sp);
    const bool again = e >= kTopAgain;
    if (!again && __uint_as_float((e >> 18) << 17) > bound) continue;
    R.set(kwCur, again ? e & ~kTopAgain : (e >> 1) & kTopIndexMask);
    next = !again && (e & 1u) ? kwInstance : kwNode;
    break;
  }
  R.set(kwSp, sp);
  return next == kwDone && rec_t < 1e30f ? kwVerify : next;
}

// One of the quantized planes of child k: 1 + q * 2^-15.
__device__ __forceinline__ uint32_t wide_q(uint32_t lo, uint32_t hi, int k) {
  return __byte_perm(k < 4 ? lo : hi, 0x3f800000u, 0x7604u | ((uint32_t)(k & 3) << 4));
}

// (near, far) plane distances of one axis of child k in one packed multiply-add.
struct Pair { float n, f; };
__device__ __forceinline__ Pair wide_planes(uint32_t n0, uint32_t n1, uint32_t f0, uint32_t f1, int k, uint64_t A,
                                            uint64_t C) {
  uint64_t q, t;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "r"(wide_q(n0, n1, k)), "r"(wide_q(f0, f1, k)));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t) : "l"(q), "l"(A), "l"(C));
  Pair p;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(p.n), "=f"(p.f) : "l"(t));
  return p;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// A wide node's boxes against a ray: t_near of every child, the sign bits of t_far - t_near
// (child k at bit k), the rest of the header.
struct WideTest { uint32_t miss, ni, nl, child; };
template <class F>
__device__ __forceinline__ WideTest wide_test(const uint4* np, float3 o, float3 rinv, float tb, F near) {
  const uint4 h = __ldg(np);
  const uint32_t child = __ldg(reinterpret_cast<const uint32_t*>(np + 1));
  const Words8 a = ldg256(np + 2);
  const uint4 c = __ldg(np + 4);
  const uint32_t e = h.w;
  constexpr float kFar = 1.000002f;
  const float Ax = __uint_as_float((e << 23) & 0x7f800000u) * rinv.x;
  const float Ay = __uint_as_float((e << 15) & 0x7f800000u) * rinv.y;
  const float Az = __uint_as_float((e << 7) & 0x7f800000u) * rinv.z;
  const float Cx = __fmaf_rn(__uint_as_float(h.x) - o.x, rinv.x, -Ax);
  const float Cy = __fmaf_rn(__uint_as_float(h.y) - o.y, rinv.y, -Ay);
  const float Cz = __fmaf_rn(__uint_as_float(h.z) - o.z, rinv.z, -Az);
  const uint64_t AX = pack2(Ax, Ax * kFar), AY = pack2(Ay, Ay * kFar), AZ = pack2(Az, Az * kFar);
  const uint64_t CX = pack2(Cx, Cx * kFar), CY = pack2(Cy, Cy * kFar), CZ = pack2(Cz, Cz * kFar);
  const bool sx = rinv.x < 0.0f, sy = rinv.y < 0.0f, sz = rinv.z < 0.0f;
  const uint32_t nx0 = sx ? a.w[2] : a.w[0], nx1 = sx ? a.w[3] : a.w[1];
  const uint32_t fx0 = sx ? a.w[0] : a.w[2], fx1 = sx ? a.w[1] : a.w[3];
  const uint32_t ny0 = sy ? a.w[6] : a.w[4], ny1 = sy ? a.w[7] : a.w[5];
  const uint32_t fy0 = sy ? a.w[4] : a.w[6], fy1 = sy ? a.w[5] : a.w[7];
  const uint32_t nz0 = sz ? c.z : c.x, nz1 = sz ? c.w : c.y;
  const uint32_t fz0 = sz ? c.x : c.z, fz1 = sz ? c.y : c.w;
  uint32_t miss = 0;
#pragma unroll
  for (int j = 7; j >= 0; --j) {
    const Pair x = wide_planes(nx0, nx1, fx0, fx1, j, AX, CX);
    const Pair y = wide_planes(ny0, ny1, fy0, fy1, j, AY, CY);
    const Pair z = wide_planes(nz0, nz1, fz0, fz1, j, AZ, CZ);
    const float tn = fmaxf(max3f(x.n, y.n, z.n), 0.0f);
    const float tf = fminf(min3f(x.f, y.f, z.f), tb);
    miss = __funnelshift_l(__float_as_uint(tf - tn), miss, 1);
    near(j, tn);
  }
  return WideTest{miss, (e >> 24) & 15u, e >> 28, child};
}

// Visit a node: in a BLAS the next child of the current (interior) group; in the TLAS
// the current one, whose children hit go on the stack, the nearest on top.
__device__ __forceinline__ uint32_t wide_node(const WideRay& R, const DevScene& S, const TraceCfg& cfg) {
  uint32_t spx = R.u(kwSp);
  const bool blas = (spx & kInBlas) != 0u;
  const float3 rinv = v3(wide_rcp(R.f(kwDX)), wide_rcp(R.f(kwDY)), wide_rcp(R.f(kwDZ)));
  uint32_t at = R.u(kwCur);
  if (blas) {
    const uint32_t grp = R.u(kwGrp), axis = (grp >> kWideIndexBits) & 3u, hits = grp >> 24;
    const float along = axis == 0u ? rinv.x : axis == 1u ? rinv.y : rinv.z;
    const uint32_t k = along < 0.0f ? 31u - __clz(hits) : __ffs(hits) - 1u;
    const uint32_t rest = grp & ~(0x1000000u << k);
    at = (grp & kWideIndexMask) + k;
    if (rest >> 24) R.stack(spx++ & 0x7fu) = rest;
  }
  float tn[8];
  const uint32_t node = blas ? at : at & kTopIndexMask;
  const uint4* np = (blas ? S.wide_blas : S.wide_tlas) + (size_t)node * (kWideNodeWords / 4);
  const WideTest w = wide_test(np, R.f3(kwOX), rinv, R.f(kwCull), [&](int k, float t) { tn[k] = t; });
  const uint32_t ih = ~w.miss & ((1u << w.ni) - 1u), lh = ~w.miss & (0xff00u >> w.nl) & 0xffu;
  if (blas) {
    const uint32_t inner = (w.child & (kWideIndexMask | (3u << kWideIndexBits))) | (ih << 24);
    if (lh) {
      if (ih) R.stack(spx++ & 0x7fu) = inner;
      uint32_t leaves = at | (3u << kWideIndexBits) | (lh << 24);
      R.set(kwCur, wide_leaf(S, leaves));
      R.set(kwGrp, leaves);
      R.set(kwSp, spx);
      return kwTriangles;
    }
    if (ih) {
      R.set(kwGrp, inner);
      R.set(kwSp, spx);
      return kwNode;
    }
    return wide_pop(R, spx);
  }
  const float rec_t = R.f(kwRecT), slack = S.wide_slack;
  const float bound = fminf(wide_bound(rec_t, kLeastSlack), R.f(kwFar));
  uint32_t hit = (ih | lh) & ~(at >> kTopIndexBits);
  uint32_t sp = spx;
  if (hit) {
    if (sp + __popc(hit) > cfg.stack_top) {
      const uint32_t rest = hit & (hit - 1u);
      if (rest) R.stack(sp++) = kTopAgain | ((rest ^ 0xffu) << kTopIndexBits) | node;
      hit ^= rest;
    }
    const uint4 ra = __ldg(np + 1), rb = __ldg(np + 5);  // references of the leaves
    const uint32_t ref[8] = {ra.x, rb.w, rb.z, rb.y, rb.x, ra.w, ra.z, ra.y};
    const uint32_t child = w.child & kWideIndexMask;
    uint32_t loose = 0;
    if (slack > kLeastSlack) {
      loose = ih & (w.child >> kTopLooseShift);
#pragma unroll
      for (int k = 0; k < 8; ++k) loose |= lh & ((ref[k] >> 31) << k);
    }
    const float less = __fdividef(1.0f, 1.0f + slack);
    float best = 3.4e38f;
    uint32_t best_e = 0, best_at = sp, e = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool inner = (uint32_t)k < w.ni;
      float at_least = tn[k];
      if (loose & (1u << k)) at_least = fmaxf((at_least - slack) * less, 0.0f);
      if ((hit & (1u << k)) && at_least <= bound) {
        e = ((__float_as_uint(at_least) >> 17) << 18) | (inner ? (child + (uint32_t)k) << 1 : (ref[k] << 1) | 1u);
        if (tn[k] < best) { best = tn[k]; best_e = e; best_at = sp; }
        R.stack(sp++) = e;
      }
    }
    if (best < 3.4e38f) {
      R.stack(best_at) = e;
      R.stack(sp - 1u) = best_e;
    }
  }
  return wide_top_pop(R, sp, bound, rec_t);
}

// The t of a triangle that ray_triangle_v may accept with t <= gate, up to two
// roundings; 1e30 when it cannot: its comparisons without the division, each with a margin
// above its rounding.
__device__ __forceinline__ float wide_candidate(float3 o, float3 d, float gate, float4 g0, float4 g1, float4 g2,
                                                const TraceCfg& cfg) {
  const float3 e1 = xyz(g1), e2 = xyz(g2);
  const float3 h = cross(d, e2);
  const float a = dot(e1, h);
  const float3 s = sub(o, xyz(g0));
  const float3 q = cross(s, e1);
  const uint32_t neg_a = __float_as_uint(a) & 0x80000000u;
  const float A = fabsf(a) * 1.000002f;
  const float U = __uint_as_float(__float_as_uint(dot(s, h)) ^ neg_a);
  const float V = __uint_as_float(__float_as_uint(dot(d, q)) ^ neg_a);
  const float t = __fdividef(__uint_as_float(__float_as_uint(dot(e2, q)) ^ neg_a), fabsf(a));
  const bool may = fabsf(a) >= cfg.eps_par && !(fminf(U, V) < -1e-30f) && !(U + V > A) &&
                   t > cfg.eps_tri * 0.99999f && t <= gate;
  return may ? t : 1e30f;
}

// The nearest of a leaf's hits by the reference's arithmetic, the first in the leaf's order of
// those at the same t: among n triangles from `first` on and, unless it is kWideRootLeaf, the earlier
// triangle `slot` of the same leaf.  kWideRootLeaf if there is none or `slot` is no such hit.  Both
// sides of a surface modelled twice lie in one leaf, and every ray onto it comes here: 720p frames
// of 40 such spheres and of the Cornell box take 2.8 and 1.5 ms; traced again the rays took 7.1 and
// 3.7, and the binary trees take 5.5 and 2.3.
static __device__ __noinline__ uint32_t wide_nearest(const DevScene& S, const TraceCfg& cfg, float3 o, float3 d,
                                                     uint32_t slot, uint32_t first, uint32_t n) {
  float best = 1e30f, t, u, v;
  uint32_t at = kWideRootLeaf;
  if (slot != kWideRootLeaf) {
    const float4* a = S.tri_bvh + (size_t)slot * 3;
    const float4 a1 = __ldg(a + 1);
    if (__float_as_uint(a1.w) != __float_as_uint(__ldg(S.tri_bvh + (size_t)first * 3 + 1).w)) return at;
    if (!ray_triangle_v(o, d, best, xyz(__ldg(a)), xyz(a1), xyz(__ldg(a + 2)), cfg, best, u, v)) return at;
    at = slot;
  }
  for (uint32_t k = 0; k < n; ++k)
    if (ray_triangle(o, d, best, S.tri_bvh + (size_t)(first + k) * 3, cfg, t, u, v)) {
      best = t;
      at = first + k;
    }
  return at;
}

// The next triangles of the current leaf: kTrisPerVisit, or two when no ray of the step has
// more left.  Leaves hold 5.8 triangles on average (BLAS leaf size 8): the 1080p sphere
// frame took 10.9 ms with two a step, 10.2 with three, 10.0 with four.
constexpr uint32_t kTrisPerVisit = 4;
__device__ __forceinline__ uint32_t wide_tri(const WideRay& R, const DevScene& S, const TraceCfg& cfg) {
  const uint32_t cur = R.u(kwCur);
  const uint32_t first = cur & kWideFirstMask, left = cur >> kWideFirstBits;
  const bool more = __any_sync(__activemask(), left > 2u);
  const float4* tp = S.tri_bvh + (size_t)first * 3;
  float4 g[kTrisPerVisit][3];
#pragma unroll
  for (uint32_t k = 0; k < kTrisPerVisit; ++k)
    if (k < 2u || more) {
      const float4* tq = k < left ? tp + 3 * k : tp;
#pragma unroll
      for (int j = 0; j < 3; ++j) g[k][j] = __ldg(tq + j);
    }
  const float3 o = R.f3(kwOX), d = R.f3(kwDX);
  const float len = R.f(kwLen), best = R.f(kwRecT), eps = R.f(kwEps);
  // (a hit beyond an occlusion query's limit and the rounding of distances hides nothing, and a
  // hit before it has its boxes verified: most shadow rays end without a candidate to
  // verify or to trace again.  512^2 x 16 spp Cornell frame 5.72 -> 5.46 ms)
  const float gate = fminf(best < 1e30f ? wide_gate(best, eps) * len : 1e30f, wide_gate(R.f(kwLimit), eps) * len);
  float ta = 1e30f, tb = 1e30f;  // the nearest candidate and the second
  uint32_t ka = 0;
#pragma unroll
  for (uint32_t k = 0; k < kTrisPerVisit; ++k)
    if (k < 2u || more) {
      const float x = wide_candidate(o, d, gate, g[k][0], g[k][1], g[k][2], cfg);
      const float t = k < left ? x : 1e30f;
      tb = fminf(tb, fmaxf(ta, t));
      ka = t < ta ? k : ka;
      ta = fminf(ta, t);
    }
  if (ta < 1e30f) {
    const float scale = __fdividef(1.0f, len);
    const float w = ta * scale;
    const uint32_t spx = R.u(kwSp), inst = (spx >> 14) & kInstMask;
    uint32_t slot = first + ka;
    const bool decided = wide_decides(R, w);  // an occlusion query's light is hidden, if this hit is verified
    // the nearest of all and the second: ambiguous within the nearest's gate
    const float second = fminf(fmaxf(w, best), tb < 1e30f ? tb * scale : 1e30f), M = wide_gate(fminf(w, best), eps);
    bool nearer = w < best;
    if (!decided && second <= M) {  // of one leaf: the reference's order is that of their slots
      const bool with = best <= M;
      if (with && (R.u(kwRecInst) & kInstMask) != inst) return kwRedo;
      const uint32_t rec = with ? R.u(kwRecSlot) : kWideRootLeaf;
      slot = wide_nearest(S, cfg, o, d, rec, first, min(left, more ? kTrisPerVisit : 2u));
      if (slot == kWideRootLeaf) return kwRedo;
      nearer = slot != rec;
    }
    if (nearer) {
      R.setf(kwRecT, fminf(w, best));
      R.set(kwRecSlot, slot);
      R.set(kwRecInst, (R.u(kwRecInst) & ~kInstMask) | inst);
      R.setf(kwCull, fminf(wide_bound(M, R.f(kwSlack)) * len, R.f(kwCull)));
    }
    if (decided) return kwVerify;
  }
  const uint32_t done = more ? kTrisPerVisit : 2u;
  if (left > done) {
    R.set(kwCur, cur + done - (done << kWideFirstBits));
    return kwTriangles;
  }
  uint32_t grp = R.u(kwGrp);
  if (grp >> 24) {
    R.set(kwCur, wide_leaf(S, grp));
    R.set(kwGrp, grp);
    return kwTriangles;
  }
  return wide_pop(R, R.u(kwSp));
}

// The object-space ray of an instance (the first columns of its record), as trace_do enters it;
// returns the length of the transformed direction.  The matrix is affine and the ray finite, so
// the position's fourth component is that of the fourth column.
__device__ __forceinline__ float wide_object_ray(const M4& w2o, float3 wo, float3 wd, float3& o, float3& d) {
  const float4 p = mul4(w2o, wo.x, wo.y, wo.z, 1.0f);
  o = v3(p.x / w2o.c3.w, p.y / w2o.c3.w, p.z / w2o.c3.w);
  const float3 dw = transform_direction(w2o, wd);
  const float len = length(dw);
  d = divs(dw, len);
  return len;
}

// The margin of distances (wide_gate) that an instance with the given record and object ray adds to
// that of the ray's origin.
__device__ __forceinline__ float wide_margin(const M4& w2o, float3 wo, float3 o, float len) {
  return fmaxf(__fdividef(1.6e-6f * max_abs3(o), len), w2o.c1.w * max_abs3(wo) + w2o.c2.w);
}

// Leave the BLAS, if in one, and enter the next instance, if one is next.
__device__ __forceinline__ uint32_t wide_instance(const WideRay& R, const DevScene& S, float3 wo, float3 wd) {
  uint32_t sp = R.u(kwSp);
  const float rec_t = R.f(kwRecT), far = R.f(kwFar);
  if (sp & kInBlas) {
    const uint32_t next =
        wide_top_pop(R, (sp >> 7) & 0x7fu, fminf(wide_bound(rec_t, kLeastSlack), far), rec_t);
    if (next == kwNode) wide_world(R, S, wo, wd, rec_t, far);
    if (next != kwInstance) return next;
    sp = R.u(kwSp);
  }
  const uint32_t inst = R.u(kwCur);
  const float4* ip = S.inst_wide + (size_t)inst * kWideInstRows;
  const M4 w2o = load_m4(ip);
  const float4 wx = __ldg(ip + 4);
  float3 o, d;
  const float len = wide_object_ray(w2o, wo, wd, o, d);
  R.set(kwSp, sp | (sp << 7) | (inst << 14) | kInBlas);
  R.setf3(kwOX, o);
  R.setf3(kwDX, d);
  R.setf(kwLen, len);
  R.setf(kwEps, fmaxf(R.f(kwEps), wide_margin(w2o, wo, o, len)));
  const float slack = fmaxf(wx.z, __fdividef(w2o.c0.w, len));
  R.setf(kwSlack, slack);
  R.setf(kwCull, (fminf(wide_bound(rec_t, slack), far) + 1e-3f * (1.0f + max_abs3(wo))) * len);
  const uint32_t root = __float_as_uint(wx.x);
  R.set(kwCur, __float_as_uint(wx.y));
  R.set(kwGrp, root);
  if (!wide_ray_ok(o, d)) return kwRedo;
  return root ? kwNode : kwTriangles;
}

// Whether a launch over scene S with the given settings (trace_stacks done) may
// take the wide traversal: no push or visit is ever dropped by the
// reference's limits, and the slacks were made for an eps_par of at least 1e-4.
__host__ __device__ inline bool wide_allowed(const TraceCfg& tc, const DevScene& S) {
  return S.wide && S.fast_slabs && tc.cull && tc.step_policy == 0u && tc.eps_par >= 0.99e-4f && tc.eps_tri >= 0.0f;
}

// The binary traversal of a ray the wide one left undecided.
static __device__ __noinline__ void wide_exact(const DevScene& S, const TraceCfg& cfg, Counters* ctr, float3 wo,
                                               float3 wd, float limit, Hit* out) {
  uint32_t stk[2 * 64 + kColdWords];
  trace_closest<false>(S, wo, wd, *out, stk, 1u, cfg, ctr, nullptr, limit);
}
__device__ __forceinline__ void wide_store(const WideRay& R, const Hit& h) {
  R.setf(kwRecT, h.t);
  R.set(kwRecInst, (R.u(kwRecInst) & ~kInstMask) | h.inst);
  R.set(kwRecSlot, h.slot);
  R.setf(kwU, h.u);
  R.setf(kwV, h.v);
}

// Verify a finished ray's candidate: kwDone, or kwRedo when it fails.  The candidate of an
// occlusion query ended early needs no exact distance; its boxes of both levels are tested
// like any other's, and are entered before the limit too, so that a hit which kept the
// reference out of them hides the light as well.  (Without the instance's box, 5 of 2.7e9
// rays of Cornell frames, past the edge of a mesh of one leaf, were answered wrongly.  Testing
// it: the 512^2 x 16 spp frame 4.96 ms before and after, 5.07 with the exact test alone.)
__device__ __forceinline__ uint32_t wide_verify(const WideRay& R, const DevScene& S, const TraceCfg& cfg, float3 wo,
                                                float3 wd) {
  const float rec_t = R.f(kwRecT);
  const bool decided = wide_decides(R, rec_t);
  Hit h;
  h.inst = R.u(kwRecInst) & kInstMask;
  const uint32_t slot = R.u(kwRecSlot);
  const float4* ip = S.inst_wide + (size_t)h.inst * kWideInstRows;
  const float4 wy = __ldg(ip + 5);
  const float4* tp = S.tri_bvh + (size_t)slot * 3;
  const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
  float3 o, d;
  const M4 w2o = load_m4(ip);
  const float len = wide_object_ray(w2o, wo, wd, o, d);
  // (the hit's own margin: kwEps may have grown since hits were looked for up to the gate, and a
  // box entered between the two gates can have let one beyond the first win)
  const float gate = wide_gate(rec_t, fmaxf(1e-6f * max_abs3(wo), wide_margin(w2o, wo, o, len))) * 0.999999f;
  const float by = decided ? (2.0f * R.f(kwLimit) - R.f(kwFar)) * 0.999999f : gate;
  float t = 0.0f;
  h.u = h.v = 0.0f;
  bool ok = ray_triangle_v(o, d, 1e30f, xyz(t0), xyz(t1), xyz(t2), cfg, t, h.u, h.v);
  const uint32_t leaf = __float_as_uint(t1.w), tleaf = __float_as_uint(wy.z);
  if (leaf != kWideRootLeaf)
    ok = ok && enters_box(o, d, S.blas_nodes + 2 * (size_t)(__float_as_uint(wy.y) + leaf), by * len);
  if (tleaf != kWideRootLeaf) ok = ok && enters_box(wo, wd, S.tlas_nodes + 2 * (size_t)tleaf, by);
  h.t = -3.0e38f;
  if (!decided) {
    const M4 o2w = load_m4(S.instances + (size_t)h.inst * 10);
    h.t = length(sub(transform_position(o2w, add(o, muls(d, t))), wo));
    ok = ok && h.t < 1e30f && h.t <= gate;
  }
  h.slot = slot - __float_as_uint(wy.x);  // within the mesh
  wide_store(R, h);
  return ok ? kwDone : kwRedo;
}

// The closest hit of a finished ray (t = -3e38 when an occlusion query ended early).
__device__ __forceinline__ Hit wide_hit(const WideRay& R) {
  Hit h = fresh_hit();
  const float t = R.f(kwRecT);
  if (t < 1e30f) {
    h.t = t;
    h.inst = R.u(kwRecInst) & kInstMask;
    h.slot = R.u(kwRecSlot);
    h.u = R.f(kwU);
    h.v = R.f(kwV);
  }
  return h;
}

// Runs a warp's pool until the items are used up and every ray is finished.  Item gives
//   scene(R)            the slot's scene,
//   ray(R, o, d, limit) its world ray (read again where it is needed: seven words less
//                       of shared memory a slot),
//   fetch(R, i)         begin item i in the slot: its class (kwDone: finished at once),
//   finish(R)           the ray is finished: kwEmpty, or kwShade (with kShades),
//   shade(R)            the item's own step: the next class.
// Each step performs the class most slots wait for (at most 32 count); rays to be traced
// again wait for kRedoAt of them, as they run alone in the warp (lane by lane they took
// 1.5 of the 7.2 ms of the 512^2 x 16 spp Cornell frame, whose boxes stand on the floor).  New items
// are fetched once kFetchAt slots are empty, or once one is and no other class has a slot.  (A
// pool full of rays to be traced again has none empty: those are traced then, so that every step
// takes a slot on.)  The warp's first kPool items are those of its number, later ones come from
// the cursor kFetchChunk at a time (an atomic takes about 2 us when every warp asks).
constexpr uint32_t kFetchAt = 16, kFetchChunk = 64, kRedoAt = 16;

template <class Item>
__device__ __forceinline__ void wide_run(Item& it, const TraceCfg& tc, uint32_t* pool, uint32_t* cursor,
                                         uint32_t n_items, Counters* ctr) {
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  uint8_t* cls = reinterpret_cast<uint8_t*>(pool + (kWideWords + tc.stack_w) * kPool);
  uint8_t* list = cls + kPool;
  reinterpret_cast<uint16_t*>(cls)[lane] = (uint16_t)(kwEmpty | (kwEmpty << 8));
  __syncwarp();
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t share = min(kPool, (n_items + warps - 1u) / warps);  // of the first, fixed items
  uint32_t at = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * share;
  uint32_t end = min(at + share, n_items);
  at = min(at, end);
  bool drained = false;  // nothing left to fetch
  while (true) {
    const uint32_t two = reinterpret_cast<const uint16_t*>(cls)[lane];
    const uint32_t c0 = two & 0xffu, c1 = two >> 8;
    // slots per class, seven bits each for the first four
    const uint32_t packed =
        __reduce_add_sync(0xffffffffu, (c0 < 4u ? 1u << (7u * c0) : 0u) + (c1 < 4u ? 1u << (7u * c1) : 0u));
    // the fullest: count << 3 | class
    const uint32_t kn = (packed & 127u) << 3, kt = ((packed >> 4) & 0x3f8u) | 1u;
    const uint32_t ki = ((packed >> 11) & 0x3f8u) | 2u, kv = ((packed >> 18) & 0x3f8u) | 3u;
    uint32_t key = max(max(kn, kt), max(ki, kv));
    const uint32_t rest = kPool - (kn >> 3) - (kt >> 3) - (ki >> 3) - (kv >> 3);
    if (Item::kShades || rest >= kFetchAt || key < 8u) {
      const uint32_t nr = __popc(__ballot_sync(0xffffffffu, c0 == kwRedo)) + __popc(__ballot_sync(0xffffffffu, c1 == kwRedo));
      uint32_t ns = 0u;
      if (Item::kShades) {
        ns = __popc(__ballot_sync(0xffffffffu, c0 == kwShade)) + __popc(__ballot_sync(0xffffffffu, c1 == kwShade));
        key = max(key, (ns << 3) | kwShade);
      }
      const uint32_t free = rest - nr - ns;
      if (!drained && (free >= kFetchAt || (key < 8u && free))) key = kwEmpty;
      else if (nr >= kRedoAt || (key < 8u && nr)) key = kwRedo;
      else if (key < 8u) break;
    }
    const uint32_t act = key & 7u;
    const uint32_t b0 = __ballot_sync(0xffffffffu, c0 == act), b1 = __ballot_sync(0xffffffffu, c1 == act);
    const uint32_t n0 = __popc(b0);
    uint32_t n = min(n0 + __popc(b1), 32u);
    const uint32_t r0 = __popc(b0 & below), r1 = n0 + __popc(b1 & below);
    if (c0 == act) list[r0] = (uint8_t)(2u * lane);
    if (c1 == act && r1 < 32u) list[r1] = (uint8_t)(2u * lane + 1u);
    uint32_t item = 0;
    if (act == kwEmpty) {
      if (at == end) {
        if (lane == 0) at = atomicAdd(cursor, kFetchChunk);
        at = warps * share + __shfl_sync(0xffffffffu, at, 0);
        end = min(at + kFetchChunk, n_items);
        if (at >= n_items || warps * share >= n_items) {
          at = end = 0u;
          drained = true;
        }
      }
      n = min(n, end - at);
      item = at + lane;
      at += n;
    }
    __syncwarp();
    if (lane < n) {
      const uint32_t slot = list[lane];
      const WideRay R{pool + slot};
      uint32_t next;
      if (act == kwNode) {
        next = wide_node(R, it.scene(R), tc);
      } else if (act == kwTriangles) {
        next = wide_tri(R, it.scene(R), tc);
      } else if (act == kwEmpty) {
        next = it.fetch(R, item);
      } else if (act == kwShade) {
        next = it.shade(R);
      } else {
        float3 wo, wd;
        float limit;
        it.ray(R, wo, wd, limit);
        if (act == kwInstance) {
          next = wide_instance(R, it.scene(R), wo, wd);
        } else if (act == kwVerify) {
          next = wide_verify(R, it.scene(R), tc, wo, wd);
        } else {
          Hit h;
          wide_exact(it.scene(R), tc, ctr, wo, wd, limit, &h);
          wide_store(R, h);
          next = kwDone;
        }
      }
      if (next == kwDone) next = it.finish(R);
      cls[slot] = (uint8_t)next;
    }
    __syncwarp();
  }
}

}  // namespace pt

// wf_common.cuh -- device helpers shared by the wavefront kernels (internal).
#pragma once
#include "wavefront.h"

namespace pt {
namespace wf {

constexpr int kWfBlock = 128;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// The persistent kernels step until this many of a warp's 32 lanes are idle,
// then refill them (every refill costs a ballot round and a queue atomic per
// warp, so refilling after every step is slower).
constexpr uint32_t kRefillAt = 8;

// Whether a persistent warp should stop stepping and refill its idle lanes.
__device__ __forceinline__ bool time_to_refill(bool busy, bool drained) {
  const uint32_t idle = __popc(__ballot_sync(0xffffffffu, !busy));
  return idle == 32u || (!drained && idle >= kRefillAt);
}

// Warp-aggregated append: every lane of the warp calls it; lanes with pred
// get consecutive slots of *counter.
__device__ __forceinline__ uint32_t warp_append(bool pred, uint32_t* counter) {
  const uint32_t mask = __ballot_sync(0xffffffffu, pred);
  if (mask == 0u) return 0xffffffffu;
  const uint32_t leader = __ffs(mask) - 1u;
  uint32_t base = 0;
  if (lane_id() == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  return pred ? base + (uint32_t)__popc(mask & ((1u << lane_id()) - 1u)) : 0xffffffffu;
}

// Persistent-kernel refill: lanes with need=true get the next queue entries
// (one atomicAdd per warp); 0xffffffff when the queue is exhausted.
__device__ __forceinline__ uint32_t warp_fetch(bool need, uint32_t* cursor, uint32_t n) {
  const uint32_t mask = __ballot_sync(0xffffffffu, need);
  if (mask == 0u) return 0xffffffffu;
  const uint32_t leader = __ffs(mask) - 1u;
  uint32_t base = 0;
  if (lane_id() == leader) base = atomicAdd(cursor, (uint32_t)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  const uint32_t idx = base + (uint32_t)__popc(mask & ((1u << lane_id()) - 1u));
  return need && idx < n ? idx : 0xffffffffu;
}

__device__ __forceinline__ void load_state(const WfBuffers& B, uint32_t p, PathState& ps) {
  const float4 a = B.s[4 * (size_t)p], b = B.s[4 * (size_t)p + 1], c = B.s[4 * (size_t)p + 2],
               d = B.s[4 * (size_t)p + 3];
  ps.o = xyz(a); ps.prev_pdf = a.w;
  ps.d = xyz(b); ps.rng = __float_as_uint(b.w);
  ps.thr = xyz(c);
  const uint32_t df = __float_as_uint(c.w);
  ps.depth = df & 0xffffffu;
  ps.flags = df >> 24;
  ps.color = xyz(d);
}
__device__ __forceinline__ void store_state(const WfBuffers& B, uint32_t p, const PathState& ps) {
  B.s[4 * (size_t)p] = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.prev_pdf);
  B.s[4 * (size_t)p + 1] = make_float4(ps.d.x, ps.d.y, ps.d.z, __uint_as_float(ps.rng));
  B.s[4 * (size_t)p + 2] = make_float4(ps.thr.x, ps.thr.y, ps.thr.z,
                                       __uint_as_float((ps.depth & 0xffffffu) | (ps.flags << 24)));
  B.s[4 * (size_t)p + 3] = make_float4(ps.color.x, ps.color.y, ps.color.z, 0.0f);
}

// The scene table in shared memory: [n entries of WfScene][traversal stacks].
__device__ __forceinline__ const WfScene* load_table(const WfScene* g, uint32_t n, uint32_t* smem) {
  WfScene* t = reinterpret_cast<WfScene*>(smem);
  const uint4* src = reinterpret_cast<const uint4*>(g);
  uint4* dst = reinterpret_cast<uint4*>(t);
  const uint32_t words = n * (uint32_t)(sizeof(WfScene) / sizeof(uint4));
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  return t;
}
__device__ __forceinline__ uint32_t* stacks_after(uint32_t* smem, uint32_t n) {
  return smem + n * (uint32_t)(sizeof(WfScene) / 4);
}
__device__ __forceinline__ uint32_t scene_of(const WfScene* t, uint32_t n, uint32_t p) {
  uint32_t lo = 0, hi = n;  // last scene with path_offset <= p
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (t[mid].path_offset <= p) lo = mid; else hi = mid;
  }
  return lo;
}

// Shadow request slot ss of path p of scene sid.
__device__ __forceinline__ void put_shadow(const WfBuffers& B, uint32_t ss, const ShadowReq& rq, uint32_t p,
                                           uint32_t sid) {
  float4* e = B.shadow + 4 * (size_t)ss;
  e[0] = make_float4(rq.o.x, rq.o.y, rq.o.z, rq.limit);
  e[1] = make_float4(rq.d.x, rq.d.y, rq.d.z, __uint_as_float(p));
  e[2] = make_float4(rq.add_vis.x, rq.add_vis.y, rq.add_vis.z, __uint_as_float(sid));
  e[3] = make_float4(rq.add_occ.x, rq.add_occ.y, rq.add_occ.z, 0.0f);
}

// The contribution of shadow request i (MODE: the estimator), whose ray's closest hit is at hit_t.
template <int MODE>
__device__ __forceinline__ void finish_shadow(const WfBuffers& B, uint32_t i, float hit_t) {
  const float4* e = B.shadow + 4 * (size_t)i;
  const float4 a = e[0], b = e[1], c = e[2], d = e[3];
  const uint32_t p = __float_as_uint(b.w);
  ShadowReq rq;
  rq.limit = a.w;
  rq.add_vis = xyz(c);
  rq.add_occ = xyz(d);
  const float4 col = B.s[4 * (size_t)p + 3];
  PathState ps;
  ps.color = xyz(col);
  path_on_shadow<MODE>(ps, rq, hit_t);
  B.s[4 * (size_t)p + 3] = make_float4(ps.color.x, ps.color.y, ps.color.z, col.w);
}

}  // namespace wf
}  // namespace pt

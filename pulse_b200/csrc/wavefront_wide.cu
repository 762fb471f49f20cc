// wavefront_wide.cu -- the wavefront's traversal launches over the eight-wide trees
// (pt_wide.cuh): every warp works on a pool of 64 rays in shared memory and performs, per
// step, one action for up to 32 of them.
//
// What bounded the binary kernels (wavefront.cu) here is issue with few lanes: one ray per
// lane, 28 of 32 busy, of which 12 to 14 share an instruction.  With the wide trees a ray takes
// 31 to 34 steps, of which 20 to 22 visit a node, 18 to 22 slots a step: the 1080p sphere
// frame 13.8 -> 8.8 ms, the 4K terrain frame 40.0 -> 24.7 ms, a million query rays 4.1 -> 1.5
// ms.  What bounds these kernels is still issue (54% of the slots with 16 warps an SM; 18
// threads an instruction in the first launch, 8.4 in the last), then the drain of each launch.
#include <atomic>

#include "pt_wide.cuh"
#include "wavefront.h"
#include "wf_common.cuh"

namespace pt {

namespace {

using namespace wf;

// Blocks of four warps resident per SM.  1080p sphere frame, at the time: three 13.0 ms,
// four 11.9; later four 9.3, five and six 10.5 (their registers spill, and the pools'
// shared memory, about 50 KB a block, leaves less L1).  A launch with 64-thread blocks takes
// the same kernels: an instance of each for it had doubled the module, whose load is part of a
// process's first frame (24 -> 16 ms; frames with such blocks take the same time).
constexpr int kWideBlocks = 4;

// The scenes of a launch: one, in the kernel's parameters (ONE: reading its pointers from
// constant memory took 2% off the 1080p frames), or the table in shared memory.
template <bool ONE>
struct Scenes {
  const WfScene& one;
  const WfScene* tab;
  uint32_t n;
  __device__ __forceinline__ const WfScene& at(uint32_t i) const { return ONE ? one : tab[i]; }
  __device__ __forceinline__ const WfScene& of(const WideRay& R) const { return ONE ? one : tab[R.u(kwRecInst) >> 20]; }
  __device__ __forceinline__ uint32_t of_path(uint32_t p) const { return ONE ? 0u : scene_of(tab, n, p); }
};

// Paths of a queue and, with SHADOW >= 0 (the estimator mode), after them the previous
// segment's shadow requests.
template <int SHADOW, bool ONE>
struct ExtendItem {
  Scenes<ONE> sc;
  const WfBuffers& B;
  const TraceCfg& tc;
  const uint32_t* q;
  uint32_t n;
  __device__ __forceinline__ const DevScene& scene(const WideRay& R) const { return sc.of(R).S; }
  __device__ __forceinline__ uint32_t fetch(const WideRay& R, uint32_t i) const {
    if (SHADOW >= 0 && i >= n) {
      const float4* e = B.shadow + 4 * (size_t)(i - n);
      const float4 a = e[0], b = e[1];
      const uint32_t sid = ONE ? 0u : __float_as_uint(e[2].w);
      R.set(kwId, (i - n) | 0x80000000u);
      return wide_begin(R, sid, sc.at(sid).S, xyz(a), xyz(b), occ_limit(tc, a.w));
    }
    const uint32_t p = q[i], sid = sc.of_path(p);
    const float4 a = B.s[4 * (size_t)p], b = B.s[4 * (size_t)p + 1];
    R.set(kwId, p);
    return wide_begin(R, sid, sc.at(sid).S, xyz(a), xyz(b), 3.0e38f);
  }
  __device__ __forceinline__ void ray(const WideRay& R, float3& o, float3& d, float& limit) const {
    const uint32_t id = R.u(kwId);
    const bool shadow = SHADOW >= 0 && (id & 0x80000000u) != 0u;
    const float4* e = shadow ? B.shadow + 4 * (size_t)(id & 0x7fffffffu) : B.s + 4 * (size_t)id;
    const float4 a = e[0], b = e[1];
    o = xyz(a);
    d = xyz(b);
    limit = shadow ? occ_limit(tc, a.w) : 3.0e38f;
  }
  __device__ __forceinline__ uint32_t finish(const WideRay& R) const {
    const uint32_t id = R.u(kwId);
    if (SHADOW >= 0 && (id & 0x80000000u)) {
      finish_shadow<SHADOW < 0 ? 0 : SHADOW>(B, id & 0x7fffffffu, R.f(kwRecT));
    } else {
      const Hit h = wide_hit(R);
      B.h0[id] = make_float4(h.t, __uint_as_float(h.inst), __uint_as_float(h.slot), h.u);
      B.h1[id] = h.v;
    }
    return kwEmpty;
  }
  static constexpr bool kShades = false;
  __device__ __forceinline__ uint32_t shade(const WideRay&) const { return kwEmpty; }
};

__device__ __forceinline__ uint32_t* warp_pool(uint32_t* smem, uint32_t n_table, const TraceCfg& tc) {
  return stacks_after(smem, n_table) + (threadIdx.x >> 5) * wide_pool_words(tc.stack_w);
}

// The scenes of a block: the table goes to shared memory unless there is one scene.
template <bool ONE>
__device__ __forceinline__ Scenes<ONE> block_scenes(const WfScene& one, const WfBuffers& B, uint32_t n_table,
                                                    uint32_t* smem) {
  return Scenes<ONE>{one, ONE ? nullptr : load_table(B.table, n_table, smem), n_table};
}

// n_table: scenes of the table (0 with ONE, then `one` is the scene).
template <int SHADOW, bool ONE>
__global__ void __launch_bounds__(kWfBlock, kWideBlocks)
    k_wide_extend(const __grid_constant__ TraceCfg tc, const __grid_constant__ WfBuffers B,
                  const __grid_constant__ WfScene one, uint32_t n_table, int qi, int sq, Counters* ctr) {
  extern __shared__ uint32_t smem[];
  const uint32_t n = B.counts[qi];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // nothing of this launch reads these: the next queue's and the next shadow requests'
    // counts, the other cursors (a launch of its own for them took 2 to 3 us a segment)
    B.counts[qi ^ 1] = 0u;
    B.counts[sq ^ 1] = 0u;
    B.counts[kCountExtend + (sq & 1 ^ 1)] = 0u;
    B.counts[kCountShadow] = 0u;
  }
  ExtendItem<SHADOW, ONE> it{block_scenes<ONE>(one, B, n_table, smem), B, tc, B.q[qi], n};
  wide_run(it, tc, warp_pool(smem, n_table, tc), B.counts + kCountExtend + (sq & 1), SHADOW >= 0 ? n + B.counts[sq] : n, ctr);
}

// The last segment's shadow requests.
template <int MODE, bool ONE>
__global__ void __launch_bounds__(kWfBlock, kWideBlocks)
    k_wide_shadow(const __grid_constant__ TraceCfg tc, const __grid_constant__ WfBuffers B,
                  const __grid_constant__ WfScene one, uint32_t n_table, int sq, Counters* ctr) {
  extern __shared__ uint32_t smem[];
  ExtendItem<MODE, ONE> it{block_scenes<ONE>(one, B, n_table, smem), B, tc, nullptr, 0u};
  wide_run(it, tc, warp_pool(smem, n_table, tc), B.counts + kCountShadow, B.counts[sq], ctr);
}

// Every path still alive, to its end: a finished ray's slot waits for its shading (or for
// its shadow ray's contribution), which is one more action of the warp.  A path's
// shadow request waits in the slot of the request array that its id names.
template <int MODE, bool ONE>
struct TailItem {
  Scenes<ONE> scs;
  const WfBuffers& B;
  const TraceCfg& tc;
  const uint32_t* q;
  __device__ __forceinline__ const DevScene& scene(const WideRay& R) const { return scs.of(R).S; }
  __device__ __forceinline__ uint32_t fetch(const WideRay& R, uint32_t i) const {
    const uint32_t p = q[i], sid = scs.of_path(p);
    const float4 a = B.s[4 * (size_t)p], b = B.s[4 * (size_t)p + 1];
    R.set(kwId, p);
    return wide_begin(R, sid, scs.at(sid).S, xyz(a), xyz(b), 3.0e38f);
  }
  __device__ __forceinline__ void ray(const WideRay& R, float3& o, float3& d, float& limit) const {
    const uint32_t id = R.u(kwId);
    const bool shadow = (id & 0x80000000u) != 0u;
    const float4* e = shadow ? B.shadow + 4 * (size_t)(id & 0x7fffffffu) : B.s + 4 * (size_t)id;
    const float4 a = e[0], b = e[1];
    o = xyz(a);
    d = xyz(b);
    limit = shadow ? occ_limit(tc, a.w) : 3.0e38f;
  }
  __device__ __forceinline__ uint32_t finish(const WideRay&) const {
    return kwShade;
  }
  static constexpr bool kShades = true;
  __device__ __forceinline__ uint32_t shade(const WideRay& R) const {
    const uint32_t id = R.u(kwId), p = id & 0x7fffffffu, sid = R.u(kwRecInst) >> 20;
    const WfScene& sc = scs.at(sid);
    PathState ps;
    load_state(B, p, ps);
    ShadowReq rq;
    rq.active = false;
    if (id & 0x80000000u) {
      const float4* e = B.shadow + 4 * (size_t)p;
      rq.limit = e[0].w;
      rq.add_vis = xyz(e[2]);
      rq.add_occ = xyz(e[3]);
      path_on_shadow<MODE>(ps, rq, R.f(kwRecT));
    } else {
      path_on_hit<MODE>(sc.S, sc.pc, ps, wide_hit(R), rq);
    }
    store_state(B, p, ps);
    if (rq.active) {
      put_shadow(B, p, rq, p, sid);
      R.set(kwId, p | 0x80000000u);
      return wide_begin(R, sid, sc.S, rq.o, rq.d, occ_limit(tc, rq.limit));
    }
    if (!(ps.flags & kAlive)) return kwEmpty;
    R.set(kwId, p);
    return wide_begin(R, sid, sc.S, ps.o, ps.d, 3.0e38f);
  }
};

template <int MODE, bool ONE>
__global__ void __launch_bounds__(kWfBlock, kWideBlocks)
    k_wide_tail(const __grid_constant__ TraceCfg tc, const __grid_constant__ WfBuffers B,
                const __grid_constant__ WfScene one, uint32_t n_table, int qi, Counters* ctr) {
  extern __shared__ uint32_t smem[];
  TailItem<MODE, ONE> it{block_scenes<ONE>(one, B, n_table, smem), B, tc, B.q[qi]};
  wide_run(it, tc, warp_pool(smem, n_table, tc), B.counts + kCountTail, B.counts[qi], ctr);
}

// The adjoint's shadow requests: visibility only.
struct AdjShadowItem {
  const DevScene& S;
  const WfBuffers& B;
  const TraceCfg& tc;
  float4* rec;
  uint32_t rows, flag;
  __device__ __forceinline__ const DevScene& scene(const WideRay&) const { return S; }
  __device__ __forceinline__ uint32_t fetch(const WideRay& R, uint32_t i) const {
    const float4 a = B.shadow[4 * (size_t)i], b = B.shadow[4 * (size_t)i + 1];
    R.set(kwId, i);
    return wide_begin(R, 0u, S, xyz(a), xyz(b), occ_limit(tc, a.w));
  }
  __device__ __forceinline__ void ray(const WideRay& R, float3& o, float3& d, float& limit) const {
    const float4* e = B.shadow + 4 * (size_t)R.u(kwId);
    const float4 a = e[0], b = e[1];
    o = xyz(a);
    d = xyz(b);
    limit = occ_limit(tc, a.w);
  }
  __device__ __forceinline__ uint32_t finish(const WideRay& R) const {
    const float4* e = B.shadow + 4 * (size_t)R.u(kwId);
    if (!(R.f(kwRecT) < e[0].w)) {
      float4* r = rec + rows * (size_t)__float_as_uint(e[1].w);
      r[3].w = __uint_as_float(__float_as_uint(r[3].w) | flag);
    }
    return kwEmpty;
  }
  static constexpr bool kShades = false;
  __device__ __forceinline__ uint32_t shade(const WideRay&) const { return kwEmpty; }
};

__global__ void __launch_bounds__(kWfBlock, kWideBlocks) k_wide_adj_shadow(const __grid_constant__ DevScene S,
                                                                           const __grid_constant__ TraceCfg tc,
                                                                           const __grid_constant__ WfBuffers B, float4* rec, uint32_t rows, uint32_t flag,
                                                                           Counters* ctr) {
  extern __shared__ uint32_t smem[];
  AdjShadowItem it{S, B, tc, rec, rows, flag};
  wide_run(it, tc, warp_pool(smem, 0u, tc), B.counts + kCountShadow, B.counts[2], ctr);
}

struct RayItem {
  const DevScene& S;
  const float* rays;
  Hit* out;
  __device__ __forceinline__ const DevScene& scene(const WideRay&) const { return S; }
  __device__ __forceinline__ uint32_t fetch(const WideRay& R, uint32_t i) const {
    const float* r = rays + 6 * (size_t)i;
    R.set(kwId, i);
    return wide_begin(R, 0u, S, v3(r[0], r[1], r[2]), v3(r[3], r[4], r[5]), 3.0e38f);
  }
  __device__ __forceinline__ void ray(const WideRay& R, float3& o, float3& d, float& limit) const {
    const float* r = rays + 6 * (size_t)R.u(kwId);
    o = v3(r[0], r[1], r[2]);
    d = v3(r[3], r[4], r[5]);
    limit = 3.0e38f;
  }
  __device__ __forceinline__ uint32_t finish(const WideRay& R) const {
    out[R.u(kwId)] = wide_hit(R);
    return kwEmpty;
  }
  static constexpr bool kShades = false;
  __device__ __forceinline__ uint32_t shade(const WideRay&) const { return kwEmpty; }
};

__global__ void __launch_bounds__(kWfBlock, kWideBlocks) k_wide_trace_rays(const __grid_constant__ DevScene S,
                                                                           const __grid_constant__ TraceCfg tc,
                                                                           const float* __restrict__ rays, uint32_t n,
                                                                           Hit* __restrict__ out, Counters* ctr,
                                                                           uint32_t* cursor) {
  extern __shared__ uint32_t smem[];
  RayItem it{S, rays, out};
  wide_run(it, tc, warp_pool(smem, 0u, tc), cursor, n, ctr);
}

// Launch shape: blocks of block threads, as many as asked for (128-thread blocks per SM,
// 0: kWideBlocks) and as fit the SM's shared memory.
struct Shape { int grid; uint32_t block; size_t smem; };
Shape shape(const TraceCfg& tc, uint32_t n_scenes, uint32_t blocks_per_sm, int sms, uint32_t block) {
  Shape g;
  g.block = block;
  g.smem = (size_t)n_scenes * sizeof(WfScene) + (size_t)wide_pool_words(tc.stack_w) * 4 * (block / 32);
  uint32_t per_sm = (blocks_per_sm ? blocks_per_sm : (uint32_t)kWideBlocks) * (kWfBlock / block);
  const uint32_t fit = (uint32_t)((227u * 1024u) / (g.smem + 1024u));
  if (per_sm > fit) per_sm = fit;
  if (per_sm < 1) per_sm = 1;
  g.grid = sms * (int)per_sm;
  return g;
}
Shape shape(const TraceCfg& tc, const WfLaunch& L) {
  return shape(tc, L.one ? 0u : L.n_scenes, L.trace_blocks_per_sm, L.sms, tc.block == 64 ? 64u : (uint32_t)kWfBlock);
}

template <typename K>
cudaError_t limit(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
}

// f(whether the launch has one scene) with that as a type.
template <typename F>
void by_scenes(bool one, F f) {
  one ? f(std::true_type{}) : f(std::false_type{});
}

}  // namespace

cudaError_t wide_prepare(int mode) {
  cudaError_t e = cudaSuccess;
  auto raise = [&](auto kernel) {
    if (e == cudaSuccess) e = limit(kernel);
  };
  for (bool one : {false, true})
    by_scenes(one, [&](auto on) {
      constexpr bool ONE = decltype(on)::value;
      raise(k_wide_extend<-1, ONE>);
      if (mode == 1) raise(k_wide_extend<1, ONE>), raise(k_wide_shadow<1, ONE>), raise(k_wide_tail<1, ONE>);
      if (mode == 2) raise(k_wide_extend<2, ONE>), raise(k_wide_shadow<2, ONE>), raise(k_wide_tail<2, ONE>);
      if (mode == 0) raise(k_wide_tail<0, ONE>);
    });
  if (mode == 2) raise(k_wide_adj_shadow);
  return e;
}

void wide_extend(int shadow, const TraceCfg& tc, const WfBuffers& B, const WfLaunch& L, int qi, int sq, Counters* ctr,
                 cudaStream_t st) {
  const Shape g = shape(tc, L);
  by_scenes(L.one != nullptr, [&](auto on) {
    constexpr bool ONE = decltype(on)::value;
    const auto k = shadow == 1 ? k_wide_extend<1, ONE> : shadow == 2 ? k_wide_extend<2, ONE> : k_wide_extend<-1, ONE>;
    k<<<g.grid, g.block, g.smem, st>>>(tc, B, ONE ? *L.one : WfScene{}, ONE ? 0u : L.n_scenes, qi, sq, ctr);
  });
}

void wide_shadow(int mode, const TraceCfg& tc, const WfBuffers& B, const WfLaunch& L, int sq, Counters* ctr,
                 cudaStream_t st) {
  const Shape g = shape(tc, L);
  by_scenes(L.one != nullptr, [&](auto on) {
    constexpr bool ONE = decltype(on)::value;
    const auto k = mode == 1 ? k_wide_shadow<1, ONE> : k_wide_shadow<2, ONE>;
    k<<<g.grid, g.block, g.smem, st>>>(tc, B, ONE ? *L.one : WfScene{}, ONE ? 0u : L.n_scenes, sq, ctr);
  });
}

void wide_tail(int mode, const TraceCfg& tc, const WfBuffers& B, const WfLaunch& L, int qi, Counters* ctr,
               cudaStream_t st) {
  const Shape g = shape(tc, L);
  by_scenes(L.one != nullptr, [&](auto on) {
    constexpr bool ONE = decltype(on)::value;
    const auto k = mode == 0 ? k_wide_tail<0, ONE> : mode == 1 ? k_wide_tail<1, ONE> : k_wide_tail<2, ONE>;
    k<<<g.grid, g.block, g.smem, st>>>(tc, B, ONE ? *L.one : WfScene{}, ONE ? 0u : L.n_scenes, qi, ctr);
  });
}

void wide_adj_shadow(const TraceCfg& tc, const DevScene& S, const WfBuffers& B, float4* rec, uint32_t rec_rows,
                     uint32_t flag, uint32_t trace_blocks, Counters* ctr, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const Shape g = shape(tc, 0u, trace_blocks, sms, kWfBlock);
  k_wide_adj_shadow<<<g.grid, g.block, g.smem, st>>>(S, tc, B, rec, rec_rows, flag, ctr);
}

cudaError_t wide_trace_rays(const DevScene& S, const TraceCfg& tc, const float* rays, uint32_t n, Hit* out,
                            Counters* ctr, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  static std::atomic<uint64_t> done{0};  // one bit per device: limit raised
  const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
  if (e == cudaSuccess && !(bit && (done.load() & bit))) {
    e = limit(k_wide_trace_rays);
    if (e == cudaSuccess && bit) done.fetch_or(bit);
  }
  uint32_t* cursor = reinterpret_cast<uint32_t*>(&ctr->pad);
  if (e == cudaSuccess) e = cudaMemsetAsync(cursor, 0, 4, st);
  if (e != cudaSuccess) return e;
  const Shape g = shape(tc, 0u, 0u, sms, kWfBlock);
  k_wide_trace_rays<<<g.grid, g.block, g.smem, st>>>(S, tc, rays, n, out, ctr, cursor);
  return cudaGetLastError();
}

}  // namespace pt

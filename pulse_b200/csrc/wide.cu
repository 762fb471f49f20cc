// wide.cu -- collapses binary BVHs into the eight-wide quantized nodes of
// pt_wide.cuh.
//
// Children are found top-down: the interior child of the largest surface area is replaced by its
// two children until there are eight.  One block walks the tree level by level
// (a thread per wide node); a wide node takes a few microseconds of dependent loads and
// 64-bit arithmetic, so the blocks of a cooperative launch share the levels of large
// trees.  The instance tree of 9 instances takes 30 us (40 with 64-bit divisions by the
// quanta).
#include <cooperative_groups.h>

#include "pt_wide.cuh"
#include "wide.cuh"

namespace wide {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
  const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
  return x * y + y * z + z * x;
}

// Where the leaf node of an element goes: an array by slot, or (instances) their records.
// A TLAS also has the instances' bounds (two float4 each) and room for those of its nodes.
struct LeafSink {
  uint32_t* by_slot;
  const uint32_t* instance_of;
  float4* records;
  const float4* bounds;
  float4* node_box;
  __device__ __forceinline__ void put(uint32_t slot, uint32_t node) const {
    if (by_slot) by_slot[slot] = node;
    else records[(size_t)instance_of[slot] * pt::kWideInstRows + 5].z = __uint_as_float(node);
  }
  // A TLAS element's reference.
  __device__ __forceinline__ uint32_t ref(uint32_t slot, uint32_t* head) const {
    const uint32_t i = instance_of[slot];
    const float slack = bounds[2 * (size_t)i].w;
    if (slack <= pt::kLeastSlack) return i;
    atomicMax(head + kSlack, __float_as_uint(slack));
    const float area = bounds[2 * (size_t)i + 1].w;
    if (area > 0.0f) atomicAdd(reinterpret_cast<float*>(head + kAreas), area);
    return i | pt::kLooseRef;
  }
};

// A BLAS leaf's reference.
__device__ uint32_t leaf_ref(uint32_t first, uint32_t count, uint32_t* head) {
  if (count > pt::kWideMaxCount || first + count > (1u << pt::kWideFirstBits)) {
    head[kBad] = 1u;
    return 0u;
  }
  return (count << pt::kWideFirstBits) | first;
}

// The boxes of a wide node's children, by slot.
struct Boxes { float lo[8][3], hi[8][3]; };

// The planes of the slots in `used` into the node's words.
__device__ void quantize(uint32_t* words, const Boxes& c, uint32_t used, uint32_t* head) {
  uint8_t* q8 = reinterpret_cast<uint8_t*>(words + 8);
  bool bad = false;
  for (int j = 0; j < 3; ++j) {
    float lo = 3e38f, hi = -3e38f;
    for (uint32_t k = 0; k < 8; ++k)
      if (used & (1u << k)) {
        if (!(fabsf(c.lo[k][j]) <= 1e9f) || !(fabsf(c.hi[k][j]) <= 1e9f) || !(c.lo[k][j] <= c.hi[k][j])) bad = true;
        lo = fminf(lo, c.lo[k][j]);
        hi = fmaxf(hi, c.hi[k][j]);
      }
    if (bad) break;
    // quanta: 2^e with the children's extent in 254 of them, and large enough
    // against the coordinates for the origin to move by 1/32 of one
    const double mag = fmax(fabs((double)lo), fabs((double)hi));
    const double need = fmax(fmax(((double)hi - lo) / 254.0, mag * 7.63e-6), 1e-30);
    int e;
    frexp(need, &e);  // need <= 2^e
    const double s = ldexp(1.0, e), inv = ldexp(1.0, -e);  // (powers of two: the products are the quotients)
    const float p = __double2float_rd((double)lo - s * (1.0 / 32.0));
    words[j] = __float_as_uint(p);
    words[3] |= (uint32_t)(e + 127 + 15) << (8 * j);
    for (uint32_t k = 0; k < 8; ++k) {
      if (!(used & (1u << k))) continue;
      const double ql = floor((c.lo[k][j] - (double)p) * inv - 1.0 / 64.0);
      const double qh = ceil((c.hi[k][j] - (double)p) * inv + 1.0 / 64.0);
      if (!(ql >= 0.0) || !(qh <= 255.0)) bad = true;
      q8[16 * j + k] = (uint8_t)ql;
      q8[16 * j + 8 + k] = (uint8_t)qh;
    }
  }
  if (bad) head[kBad] = 1u;
}

__device__ __forceinline__ uint32_t used_slots(uint32_t ni, uint32_t nl) {
  return ((1u << ni) - 1u) | ((0xff00u >> nl) & 0xffu);
}

// The wide node of binary node b (interior).  A TLAS leaf of several instances is as
// many children, and the planes come later (fit_node).
__device__ void make_node(const float4* __restrict__ nodes, uint32_t b, uint32_t* out, const LeafSink& leaf_of,
                          uint32_t* queue, uint32_t* head) {
  uint32_t c[8], mult[8];  // children; places each takes
  float area[8];           // below 0: not to be opened
  uint32_t n = 0, places = 0;
  const bool tlas = leaf_of.instance_of != nullptr;
  auto places_of = [&](uint32_t node) {
    const uint32_t count = __float_as_uint(nodes[2 * (size_t)node + 1].w);
    return tlas && count ? count : 1u;
  };
  auto put = [&](uint32_t k, uint32_t node) {
    const float4 lo = nodes[2 * (size_t)node], hi = nodes[2 * (size_t)node + 1];
    c[k] = node;
    mult[k] = places_of(node);
    area[k] = __float_as_uint(hi.w) ? -1.0f : fmaxf(half_area(lo, hi), 0.0f);
    places += mult[k];
  };
  const uint32_t first = __float_as_uint(nodes[2 * (size_t)b].w);
  put(n++, first);
  put(n++, first + 1);
  if (places > 8) {
    head[kBad] = 1u;
    return;
  }
  while (places < 8) {
    int best = -1;
    float most = -0.5f;
    for (uint32_t k = 0; k < n; ++k)
      if (area[k] > most) { most = area[k]; best = (int)k; }
    if (best < 0) break;
    const uint32_t a = __float_as_uint(nodes[2 * (size_t)c[best]].w);
    if (places - 1 + places_of(a) + places_of(a + 1) > 8) {
      area[best] = -1.0f;
      continue;
    }
    places -= 1;
    put((uint32_t)best, a);
    put(n++, a + 1);
  }
  uint32_t words[pt::kWideNodeWords];
  for (uint32_t k = 0; k < pt::kWideNodeWords; ++k) words[k] = 0u;
  // slots: interior children sorted along the axis of their centres' largest spread, leaves from 7 down
  Boxes box;
  uint32_t inner[8], ni = 0, nl = 0;
  float mid[8][3], cmin[3] = {3e38f, 3e38f, 3e38f}, cmax[3] = {-3e38f, -3e38f, -3e38f};
  auto set_box = [&](uint32_t slot, uint32_t node) {
    const float4 a = nodes[2 * (size_t)node], z = nodes[2 * (size_t)node + 1];
    box.lo[slot][0] = a.x, box.lo[slot][1] = a.y, box.lo[slot][2] = a.z;
    box.hi[slot][0] = z.x, box.hi[slot][1] = z.y, box.hi[slot][2] = z.z;
  };
  for (uint32_t k = 0; k < n; ++k) {
    const float4 a = nodes[2 * (size_t)c[k]], z = nodes[2 * (size_t)c[k] + 1];
    const uint32_t start = __float_as_uint(a.w), count = __float_as_uint(z.w);
    if (count) {
      for (uint32_t i = 0; i < count; ++i) leaf_of.put(start + i, c[k]);
      for (uint32_t i = 0; i < mult[k]; ++i) {
        set_box(7u - nl, c[k]);
        words[pt::wide_ref_word(nl++)] = tlas ? leaf_of.ref(start + i, head) : leaf_ref(start, count, head);
      }
      continue;
    }
    mid[k][0] = a.x + z.x, mid[k][1] = a.y + z.y, mid[k][2] = a.z + z.z;
    for (int j = 0; j < 3; ++j) {
      cmin[j] = fminf(cmin[j], mid[k][j]);
      cmax[j] = fmaxf(cmax[j], mid[k][j]);
    }
    inner[ni++] = k;
  }
  uint32_t axis = 0;
  for (uint32_t j = 1; j < 3; ++j)
    if (cmax[j] - cmin[j] > cmax[axis] - cmin[axis]) axis = j;
  for (uint32_t i = 1; i < ni; ++i) {  // insertion sort
    const uint32_t k = inner[i];
    uint32_t j = i;
    for (; j > 0 && mid[inner[j - 1]][axis] > mid[k][axis]; --j) inner[j] = inner[j - 1];
    inner[j] = k;
  }
  words[3] = (ni << 24) | (nl << 28);
  if (ni) {
    const uint32_t at = atomicAdd(head + kCount, ni);
    if (at + ni >= (1u << pt::kWideIndexBits)) head[kBad] = 1u;
    words[4] = at | (axis << pt::kWideIndexBits);
    for (uint32_t i = 0; i < ni; ++i) {
      set_box(i, c[inner[i]]);
      queue[at + i] = c[inner[i]];
    }
  }
  if (!tlas) quantize(words, box, used_slots(ni, nl), head);
  for (uint32_t k = 0; k < pt::kWideNodeWords; ++k) out[k] = words[k];
}

// A TLAS that is one leaf: a node of its instances.
__device__ void make_root_leaf(uint32_t start, uint32_t count, uint32_t* out, const LeafSink& leaf_of,
                               uint32_t* head) {
  if (count > 8) {
    head[kBad] = 1u;
    return;
  }
  for (uint32_t k = 0; k < pt::kWideNodeWords; ++k) out[k] = 0u;
  out[3] = count << 28;
  for (uint32_t i = 0; i < count; ++i) {
    leaf_of.put(start + i, pt::kWideRootLeaf);
    out[pt::wide_ref_word(i)] = leaf_of.ref(start + i, head);
  }
}

// The planes of TLAS node i from its instances' bounds and its interior children's
// boxes (made before it), its interior children that hold a loose instance, and its own box (and
// in the first w whether it holds one).
__device__ void fit_node(uint32_t i, uint32_t* out, const LeafSink& leaf_of, uint32_t* head) {
  uint32_t* w = out + (size_t)i * pt::kWideNodeWords;
  const uint32_t ni = (w[3] >> 24) & 15u, nl = w[3] >> 28, used = used_slots(ni, nl);
  Boxes box;
  float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
  uint32_t loose = 0;
  for (uint32_t k = 0; k < 8; ++k) {
    if (!(used & (1u << k))) continue;
    const float4* b = k < ni ? leaf_of.node_box + 2 * (size_t)((w[4] & pt::kWideIndexMask) + k)
                             : leaf_of.bounds + 2 * (size_t)(w[pt::wide_ref_word(7u - k)] & ~pt::kLooseRef);
    const float4 a = __ldcg(b), z = __ldcg(b + 1);
    if (a.w > pt::kLeastSlack) loose |= 1u << k;
    box.lo[k][0] = a.x, box.lo[k][1] = a.y, box.lo[k][2] = a.z;
    box.hi[k][0] = z.x, box.hi[k][1] = z.y, box.hi[k][2] = z.z;
    for (int j = 0; j < 3; ++j) {
      lo[j] = fminf(lo[j], box.lo[k][j]);
      hi[j] = fmaxf(hi[j], box.hi[k][j]);
    }
  }
  if (ni) w[4] |= (loose & ((1u << ni) - 1u)) << pt::kTopLooseShift;
  leaf_of.node_box[2 * (size_t)i] = make_float4(lo[0], lo[1], lo[2], loose ? 1.0f : 0.0f);
  leaf_of.node_box[2 * (size_t)i + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
  if (i == 0) head[kRootArea] = __float_as_uint(half_area(leaf_of.node_box[0], leaf_of.node_box[1]));
  quantize(w, box, used, head);
}

constexpr uint32_t kMaxLevels = 64;  // of a TLAS whose nodes are fitted

template <bool GRID>
__global__ void __launch_bounds__(kBlock) k_collapse(const float4* __restrict__ nodes,
                                                     const uint32_t* __restrict__ meta, uint4* out, LeafSink leaf_of,
                                                     uint32_t* queue, uint32_t* head) {
  auto sync = [] {
    if (GRID) {
      cooperative_groups::this_grid().sync();
    } else {
      __threadfence();
      __syncthreads();
    }
  };
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  if (meta && (meta[2] != 0u || meta[0] == 0u)) {
    if (tid == 0) head[kBad] = 1u;
    return;
  }
  const float4 rlo = nodes[0], rhi = nodes[1];
  const uint32_t count = __float_as_uint(rhi.w);
  if (tid == 0) {
    const uint32_t start = __float_as_uint(rlo.w);
    const bool tlas = leaf_of.instance_of != nullptr;
    head[kBad] = 0u;
    if (tlas) head[kSlack] = head[kAreas] = 0u;
    head[kLevels] = count && tlas ? 1u : 0u;
    head[kRoot] = count && !tlas ? leaf_ref(start, count, head) : 0u;
    queue[0] = 0u;
    *(volatile uint32_t*)(head + kCount) = count && !tlas ? 0u : 1u;
    if (count && tlas) {
      make_root_leaf(start, count, reinterpret_cast<uint32_t*>(out), leaf_of, head);
      if (count <= 8) fit_node(0u, reinterpret_cast<uint32_t*>(out), leaf_of, head);
    } else {
      for (uint32_t i = 0; i < count; ++i) leaf_of.put(start + i, pt::kWideRootLeaf);
    }
  }
  if (count) return;  // the tree is one leaf
  __shared__ uint32_t level_at[kMaxLevels + 1];  // (each block its own: the same values)
  sync();
  uint32_t begin = 0, levels = 0;
  while (true) {
    const uint32_t end = *(volatile uint32_t*)(head + kCount);
    if (begin == end) break;
    if (threadIdx.x == 0 && levels < kMaxLevels) level_at[levels] = begin;
    ++levels;
    sync();  // every thread has read the count
    for (uint32_t i = begin + tid; i < end; i += stride)
      make_node(nodes, *(volatile uint32_t*)(queue + i), reinterpret_cast<uint32_t*>(out) + (size_t)i * pt::kWideNodeWords,
                leaf_of, queue, head);
    sync();
    begin = end;
  }
  if (tid == 0) head[kLevels] = levels;
  if (!leaf_of.instance_of) return;
  // TLAS: bottom-up, the deepest level first.  Fitting a box that is out of range sets kBad too,
  // so every thread has read it before the first one fits: all leave here, or all meet at every
  // barrier below.
  const bool bad = levels >= kMaxLevels || *(volatile uint32_t*)(head + kBad);
  sync();
  if (bad) {
    if (tid == 0) head[kBad] = 1u;
    return;
  }
  for (uint32_t l = levels; l-- > 0;) {
    const uint32_t from = level_at[l], to = l + 1 < levels ? level_at[l + 1] : begin;
    for (uint32_t i = from + tid; i < to; i += stride) fit_node(i, reinterpret_cast<uint32_t*>(out), leaf_of, head);
    sync();
  }
}

// Boxes around a mesh for its instances' bounds: those of the root's children's
// children (dequantized; kHullBoxes, unused ones inverted).  One block of 64 threads.
__global__ void __launch_bounds__(64) k_hull(const uint32_t* __restrict__ wide_nodes, uint32_t n_wide,
                                             const float4* __restrict__ nodes, float4* hull) {
  const uint32_t t = threadIdx.x, k = t >> 3, j = t & 7u;
  float4 lo = make_float4(3e38f, 3e38f, 3e38f, 0.0f), hi = make_float4(-3e38f, -3e38f, -3e38f, 0.0f);
  auto box_of = [&](uint32_t node, uint32_t slot) {
    const uint32_t* w = wide_nodes + (size_t)node * pt::kWideNodeWords;
    const uint8_t* q = reinterpret_cast<const uint8_t*>(w + 8);
    float l[3], h[3];
    for (int a = 0; a < 3; ++a) {
      const float p = __uint_as_float(w[a]), s = ldexpf(1.0f, (int)((w[3] >> (8 * a)) & 255u) - 127 - 15);
      l[a] = p + q[16 * a + slot] * s;
      h[a] = p + q[16 * a + 8 + slot] * s;
    }
    lo = make_float4(l[0], l[1], l[2], 0.0f);
    hi = make_float4(h[0], h[1], h[2], 0.0f);
  };
  if (n_wide == 0u) {
    if (t == 0u) lo = nodes[0], hi = nodes[1];
  } else {
    const uint32_t h = wide_nodes[3], ni = (h >> 24) & 15u, nl = h >> 28;
    if (k < ni) {
      const uint32_t child = (wide_nodes[4] & pt::kWideIndexMask) + k, c = wide_nodes[(size_t)child * pt::kWideNodeWords + 3];
      if (used_slots((c >> 24) & 15u, c >> 28) & (1u << j)) box_of(child, j);
    } else if (j == 0u && (used_slots(ni, nl) & (1u << k))) {
      box_of(0u, k);
    }
  }
  hull[2 * t] = lo;
  hull[2 * t + 1] = hi;
}

__global__ void __launch_bounds__(kBlock) k_relocate(const uint32_t* __restrict__ in, uint32_t n, uint32_t node_add,
                                                     uint32_t slot_add, uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t* a = in + (size_t)i * pt::kWideNodeWords;
  uint32_t* b = out + (size_t)i * pt::kWideNodeWords;
  uint32_t w[pt::kWideNodeWords];
  for (uint32_t k = 0; k < pt::kWideNodeWords; ++k) w[k] = a[k];
  const uint32_t ni = (w[3] >> 24) & 15u, nl = w[3] >> 28;
  if (ni) w[4] += node_add;
  for (uint32_t r = 0; r < nl; ++r) w[pt::wide_ref_word(r)] += slot_add;
  for (uint32_t k = 0; k < pt::kWideNodeWords; ++k) b[k] = w[k];
}

// How far before its box the computed t of a hit may lie, for a ray of any direction that
// passes the test's |a| >= eps_par: (t + L) * slack(triangle), L the longer edge.  First-order
// rounding analysis of ray_triangle_v (u = 2^-24; products, sums and the edges' three-term
// products bounded by permanents of the absolute values): t, u and v are off by at most
// 27 u (t + L) |e1||e2| / |a| along the plane.  With edges that leave a plane of two axes by at
// most e (its normal's component n, S = |e1||e2| / |n|), products with the third axis shrink
// with e and the bound is u (t + L) (35 S + e L (100 S + 106) / |a|): a triangle that lies in
// such a plane, like a wall or a floor, is exact to roundings at any size.  Both constants are
// raised for the second order, which needs slack < 0.5; beyond there is no bound.
__device__ __forceinline__ float triangle_slack(float3 e1, float3 e2, float l1, float l2) {
  constexpr float kU = 5.9604645e-8f, kEps = 0.99e-4f;
  const float x1[3] = {e1.x, e1.y, e1.z}, x2[3] = {e2.x, e2.y, e2.z};
  const float area = l1 * l2, longer = fmaxf(l1, l2);
  float k = 32.0f * area / kEps;
  for (int i = 0; i < 3; ++i) {
    const int a = (i + 1) % 3, b = (i + 2) % 3;
    const float off = fmaxf(fabsf(x1[i]), fabsf(x2[i]));
    const float s = area / fabsf(x1[a] * x2[b] - x1[b] * x2[a]);
    k = fminf(k, 40.0f * s + off * longer * (110.0f * s + 120.0f) / kEps);  // (NaN: the general bound)
  }
  return kU * k;
}

__global__ void __launch_bounds__(kBlock) k_leaf_area(const float4* __restrict__ nodes, uint32_t n, uint32_t* head) {
  float area = 0.0f;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 lo = nodes[2 * (size_t)i], hi = nodes[2 * (size_t)i + 1];
    if (__float_as_uint(hi.w)) area += half_area(lo, hi);
    if (i == 0u) head[kRootArea] = __float_as_uint(half_area(lo, hi));
  }
  for (int off = 16; off > 0; off >>= 1) area += __shfl_xor_sync(0xffffffffu, area, off);
  if ((threadIdx.x & 31) == 0) atomicAdd(reinterpret_cast<float*>(head + kAreas), area);
}

__global__ void __launch_bounds__(kBlock) k_extents(const float4* __restrict__ prims, uint32_t n, uint32_t* head) {
  float rel = 0.0f, abs = 0.0f;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float3 p0 = pt::xyz(prims[3 * (size_t)i]), p1 = pt::xyz(prims[3 * (size_t)i + 1]),
                 p2 = pt::xyz(prims[3 * (size_t)i + 2]);
    const float3 e1 = pt::sub(p1, p0), e2 = pt::sub(p2, p0);
    const float l1 = pt::length(e1), l2 = pt::length(e2);
    // a NaN vertex cannot be hit: its triangle does not count
    const float s = triangle_slack(e1, e2, l1, l2);
    rel = fmaxf(rel, s);
    abs = fmaxf(abs, s * fmaxf(l1, l2));
  }
  const uint32_t rm = __reduce_max_sync(0xffffffffu, __float_as_uint(rel));
  const uint32_t am = __reduce_max_sync(0xffffffffu, __float_as_uint(abs));
  if ((threadIdx.x & 31) == 0) {
    atomicMax(head + kSlack, rm);
    atomicMax(head + kSlackAbs, am);
  }
}

}  // namespace

namespace {
cudaError_t launch(const float4* nodes, uint32_t n_nodes, const uint32_t* meta, uint4* out, LeafSink leaf_of,
                   uint32_t* queue, uint32_t* head, cudaStream_t st) {
  // One block up to 16k nodes (every per-frame instance tree of the scenes here): its
  // levels cost a block barrier, and it needs no co-residency with a frame's kernels.
  if (n_nodes <= 16384u) {
    k_collapse<false><<<1, kBlock, 0, st>>>(nodes, meta, out, leaf_of, queue, head);
    return cudaGetLastError();
  }
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  void* args[] = {&nodes, &meta, &out, &leaf_of, &queue, &head};
  return cudaLaunchCooperativeKernel((const void*)k_collapse<true>, dim3((unsigned)sms), dim3(kBlock), args, 0, st);
}
}  // namespace

cudaError_t collapse(const float4* nodes, uint32_t n_nodes, uint4* out, uint32_t* leaf_of, uint32_t* queue,
                     uint32_t* head, cudaStream_t st) {
  return launch(nodes, n_nodes, nullptr, out, LeafSink{leaf_of, nullptr, nullptr, nullptr, nullptr}, queue, head, st);
}

cudaError_t collapse_tlas(const float4* nodes, uint32_t n_nodes, const uint32_t* meta, const uint32_t* instance_of,
                          float4* records, const float4* bounds, float4* node_box, uint4* out, uint32_t* queue,
                          uint32_t* head, cudaStream_t st) {
  return launch(nodes, n_nodes, meta, out, LeafSink{nullptr, instance_of, records, bounds, node_box}, queue, head, st);
}

cudaError_t hull(const uint4* wide_nodes, uint32_t n_wide, const float4* nodes, float4* out, cudaStream_t st) {
  k_hull<<<1, kHullBoxes, 0, st>>>(reinterpret_cast<const uint32_t*>(wide_nodes), n_wide, nodes, out);
  return cudaGetLastError();
}

cudaError_t relocate(const uint32_t* nodes, uint32_t n, uint32_t node_add, uint32_t slot_add, uint32_t* out,
                     cudaStream_t st) {
  if (!n) return cudaSuccess;
  k_relocate<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(nodes, n, node_add, slot_add, out);
  return cudaGetLastError();
}

cudaError_t leaf_area(const float4* nodes, uint32_t n_nodes, uint32_t* head, cudaStream_t st) {
  if (!n_nodes) return cudaSuccess;
  const uint32_t blocks = (n_nodes + kBlock - 1) / kBlock;
  k_leaf_area<<<blocks < 1184u ? blocks : 1184u, kBlock, 0, st>>>(nodes, n_nodes, head);
  return cudaGetLastError();
}

cudaError_t extents(const float4* prims, uint32_t n, uint32_t* head, cudaStream_t st) {
  if (!n) return cudaSuccess;
  const uint32_t blocks = (n + kBlock - 1) / kBlock;
  k_extents<<<blocks < 1184u ? blocks : 1184u, kBlock, 0, st>>>(prims, n, head);
  return cudaGetLastError();
}

}  // namespace wide

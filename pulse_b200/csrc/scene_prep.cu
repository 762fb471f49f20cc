// scene_prep.cu -- scene preparation kernels (see scene_prep.cuh).
#include <cfloat>

#include "pt_math.cuh"
#include "pt_wide.cuh"
#include "scene_prep.cuh"

namespace prep {

using namespace pt;

namespace {

__global__ void k_soup(const float* __restrict__ pos, const float* __restrict__ nrm, const float* __restrict__ uv,
                       const uint32_t* __restrict__ idx, uint32_t ntris, float4* prims, float4* tdata) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntris) return;
  const uint32_t v[3] = {idx[3 * t], idx[3 * t + 1], idx[3 * t + 2]};
  for (int k = 0; k < 3; ++k) {
    prims[3 * t + k] = make_float4(pos[3 * v[k]], pos[3 * v[k] + 1], pos[3 * v[k] + 2], 0.0f);
    tdata[5 * t + k] = make_float4(nrm[3 * v[k]], nrm[3 * v[k] + 1], nrm[3 * v[k] + 2], 0.0f);
  }
  tdata[5 * t + 3] = make_float4(uv[2 * v[0]], uv[2 * v[0] + 1], uv[2 * v[1]], uv[2 * v[1] + 1]);
  tdata[5 * t + 4] = make_float4(uv[2 * v[2]], uv[2 * v[2] + 1], 0.0f, 0.0f);
}

// 4x4 inverse by the adjugate from 2x2 minors (D. Eberly, "The Laplace
// Expansion Theorem: Computing the Determinants and Inverses of Matrices").
// Same operation order as the CPU restatement (glam's own order is not
// available offline).
__device__ void inverse4(const float* src, float* dst) {
#define A(r, c) src[(c)*4 + (r)]
  const float s0 = A(0, 0) * A(1, 1) - A(1, 0) * A(0, 1);
  const float s1 = A(0, 0) * A(1, 2) - A(1, 0) * A(0, 2);
  const float s2 = A(0, 0) * A(1, 3) - A(1, 0) * A(0, 3);
  const float s3 = A(0, 1) * A(1, 2) - A(1, 1) * A(0, 2);
  const float s4 = A(0, 1) * A(1, 3) - A(1, 1) * A(0, 3);
  const float s5 = A(0, 2) * A(1, 3) - A(1, 2) * A(0, 3);
  const float c5 = A(2, 2) * A(3, 3) - A(3, 2) * A(2, 3);
  const float c4 = A(2, 1) * A(3, 3) - A(3, 1) * A(2, 3);
  const float c3 = A(2, 1) * A(3, 2) - A(3, 1) * A(2, 2);
  const float c2 = A(2, 0) * A(3, 3) - A(3, 0) * A(2, 3);
  const float c1 = A(2, 0) * A(3, 2) - A(3, 0) * A(2, 2);
  const float c0 = A(2, 0) * A(3, 1) - A(3, 0) * A(2, 1);
  const float det = s0 * c5 - s1 * c4 + s2 * c3 + s3 * c2 - s4 * c1 + s5 * c0;
  const float id = 1.0f / det;
  float b[4][4];
  b[0][0] = (A(1, 1) * c5 - A(1, 2) * c4 + A(1, 3) * c3) * id;
  b[0][1] = (-A(0, 1) * c5 + A(0, 2) * c4 - A(0, 3) * c3) * id;
  b[0][2] = (A(3, 1) * s5 - A(3, 2) * s4 + A(3, 3) * s3) * id;
  b[0][3] = (-A(2, 1) * s5 + A(2, 2) * s4 - A(2, 3) * s3) * id;
  b[1][0] = (-A(1, 0) * c5 + A(1, 2) * c2 - A(1, 3) * c1) * id;
  b[1][1] = (A(0, 0) * c5 - A(0, 2) * c2 + A(0, 3) * c1) * id;
  b[1][2] = (-A(3, 0) * s5 + A(3, 2) * s2 - A(3, 3) * s1) * id;
  b[1][3] = (A(2, 0) * s5 - A(2, 2) * s2 + A(2, 3) * s1) * id;
  b[2][0] = (A(1, 0) * c4 - A(1, 1) * c2 + A(1, 3) * c0) * id;
  b[2][1] = (-A(0, 0) * c4 + A(0, 1) * c2 - A(0, 3) * c0) * id;
  b[2][2] = (A(3, 0) * s4 - A(3, 1) * s2 + A(3, 3) * s0) * id;
  b[2][3] = (-A(2, 0) * s4 + A(2, 1) * s2 - A(2, 3) * s0) * id;
  b[3][0] = (-A(1, 0) * c3 + A(1, 1) * c1 - A(1, 2) * c0) * id;
  b[3][1] = (A(0, 0) * c3 - A(0, 1) * c1 + A(0, 2) * c0) * id;
  b[3][2] = (-A(3, 0) * s3 + A(3, 1) * s1 - A(3, 2) * s0) * id;
  b[3][3] = (A(2, 0) * s3 - A(2, 1) * s1 + A(2, 2) * s0) * id;
#undef A
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) dst[c * 4 + r] = b[r][c];
}

__global__ void k_instances(const InstanceIn* __restrict__ in, uint32_t n, const float4* __restrict__ blas_nodes,
                            float4* inst_out, float* bounds9, float4* wide_out,
                            const uint32_t* __restrict__ slot) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const InstanceIn x = in[j];
  const uint32_t i = slot ? slot[j] : j;
  float inv[16];
  inverse4(x.object_world, inv);
  float4* o = inst_out + (size_t)i * 10;
  for (int c = 0; c < 4; ++c) {
    o[c] = make_float4(x.object_world[4 * c], x.object_world[4 * c + 1], x.object_world[4 * c + 2], x.object_world[4 * c + 3]);
    o[4 + c] = make_float4(inv[4 * c], inv[4 * c + 1], inv[4 * c + 2], inv[4 * c + 3]);
  }
  o[8] = make_float4(__uint_as_float(x.triangle_offset), __uint_as_float(x.triangle_count),
                     __uint_as_float(x.index_offset), __uint_as_float(x.node_offset));
  o[9] = make_float4(__uint_as_float(x.material_index), 0.0f, 0.0f, 0.0f);
  if (wide_out) {  // the wide traversal's record (pt_wide.cuh); its TLAS leaf comes with the tree
    float4* wo = wide_out + (size_t)i * kWideInstRows;
    for (int c = 0; c < 4; ++c) wo[c] = make_float4(inv[4 * c], inv[4 * c + 1], inv[4 * c + 2], inv[4 * c + 3]);
    wo[0].w = x.wide_slack_abs;
    wo[4] = make_float4(__uint_as_float(x.wide_root), __uint_as_float(x.wide_leaf), x.wide_slack, __uint_as_float(x.hull));
    wo[5] = make_float4(__uint_as_float(x.index_offset), __uint_as_float(x.node_offset),
                        __uint_as_float(kWideRootLeaf), x.wide_leaves);
  }
  // World bounds of the root box (src/scene/mod.rs:625-658).
  const float4 lo = blas_nodes[2 * (size_t)x.node_offset], hi = blas_nodes[2 * (size_t)x.node_offset + 1];
  const M4 m{o[0], o[1], o[2], o[3]};
  const float3 corners[8] = {v3(lo.x, lo.y, lo.z), v3(hi.x, lo.y, lo.z), v3(lo.x, hi.y, lo.z), v3(lo.x, lo.y, hi.z),
                             v3(hi.x, hi.y, lo.z), v3(lo.x, hi.y, hi.z), v3(hi.x, lo.y, hi.z), v3(hi.x, hi.y, hi.z)};
  float3 wmin = v3(FLT_MAX, FLT_MAX, FLT_MAX), wmax = v3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
  float3 tc[8];
  for (int c = 0; c < 8; ++c) tc[c] = transform_position(m, corners[c]);
  for (int c = 0; c < 8; ++c) wmin = vmin(wmin, tc[c]);
  for (int c = 0; c < 8; ++c) wmax = vmax(wmax, tc[c]);
  const float3 center = add(wmin, muls(sub(wmax, wmin), 0.5f));
  float* b = bounds9 + (size_t)i * 9;
  b[0] = wmin.x; b[1] = wmin.y; b[2] = wmin.z;
  b[3] = wmax.x; b[4] = wmax.y; b[5] = wmax.z;
  b[6] = center.x; b[7] = center.y; b[8] = center.z;
}

// Row i of an instance's matrices: what the rounding of a point's way into the object's space and
// back, in units of 2^-24, multiplies the largest coordinate by (x), and adds to it (y); the
// inverse's own error is in both.  x is at most 3 and the inverse's error at most 5 for rotations
// and scales along the object's axes.
__device__ __forceinline__ float2 way_back(const M4& m, const M4& w, int i, float& defect, float& offset) {
  auto at = [](float4 c, int k) { return k == 0 ? c.x : k == 1 ? c.y : c.z; };
  const float4 oc[3] = {m.c0, m.c1, m.c2};
  const float4 wc[4] = {w.c0, w.c1, w.c2, w.c3};
  const double by = 1.0 / w.c3.w;
  float2 r = make_float2(0.0f, fabsf(at(m.c3, i)));
  defect = offset = 0.0f;
  for (int j = 0; j < 4; ++j) {
    double sum = j == 3 ? (double)at(m.c3, i) : j == i ? -1.0 : 0.0;
    float abs = 0.0f;
    for (int k = 0; k < 3; ++k) {
      sum += (double)at(oc[k], i) * at(wc[j], k) * by;
      abs += fabsf(at(oc[k], i) * at(wc[j], k));
    }
    if (j < 3) r.x += abs, defect += (float)fabs(sum);
    else r.y += abs, offset = (float)fabs(sum);
  }
  return r;
}

// One warp per instance, two hull boxes per lane.  A rotated mesh fills about half the
// cross-section of the box around its root box's corners: the rays of the 1080p sphere
// frame enter 4.5 instances instead of 6.9 (frame 11.9 -> 10.9 ms).
// The bounds are widened by four roundings of the transform's and the ray's coordinates
// times their amplification (the product of the matrix's and its inverse's largest
// entries); where that exceeds 8 the reference's bounds stay.
__global__ void __launch_bounds__(256) k_tight_bounds(uint32_t n, const float4* __restrict__ instances,
                                                      float4* inst_wide, const float* __restrict__ bounds9,
                                                      const float4* __restrict__ hulls, float4* out) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (i >= n) return;
  const M4 m = load_m4(instances + (size_t)i * 10), w = load_m4(instances + (size_t)i * 10 + 4);
  const float4* h = hulls + (size_t)__float_as_uint(inst_wide[(size_t)i * kWideInstRows + 4].w) * 128;
  float3 lo = v3(3e38f, 3e38f, 3e38f), hi = v3(-3e38f, -3e38f, -3e38f);
  for (uint32_t k = lane; k < 64u; k += 32u) {
    const float4 a = __ldg(h + 2 * k), z = __ldg(h + 2 * k + 1);
    if (!(a.x <= z.x)) continue;
    for (int c = 0; c < 8; ++c) {
      const float3 p = transform_position(m, v3(c & 1 ? z.x : a.x, c & 2 ? z.y : a.y, c & 4 ? z.z : a.z));
      lo = v3(fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z));
      hi = v3(fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z));
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    lo = v3(fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, off)), fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, off)),
            fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, off)));
    hi = v3(fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, off)), fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, off)),
            fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, off)));
  }
  // Distances of hits of a sheared instance are compared with those of others with its own
  // margin (twice the error of the way back, of a distance and of a direction): per largest
  // coordinate of the ray's origin (e1), and to add (e0).  Rotations and scales along the
  // object's axes have the traversal's (wide_gate).
  constexpr float kU = 5.9604645e-8f;
  float defect, offset;
  const float2 row = way_back(m, w, lane < 2u ? (int)lane : 2, defect, offset);
  const float* b = bounds9 + (size_t)i * 9;
  float extent = 0.0f;
  for (int k = 0; k < 6; ++k) extent = fmaxf(extent, fabsf(b[k]));
  const bool own = row.x > 3.1f || defect > 8.0f * kU || offset > 6.0f * kU * row.y;
  const float far = 3.5f * (defect + 20.0f * kU * row.x);
  float e1 = 5.5f * defect + 86.0f * kU * row.x, e0 = 2.0f * offset + 20.0f * kU * row.y + far * extent;
  if (!__any_sync(0xffffffffu, own)) e1 = e0 = 0.0f;
  for (int off = 2; off > 0; off >>= 1) {
    e1 = fmaxf(e1, __shfl_xor_sync(0xffffffffu, e1, off));
    e0 = fmaxf(e0, __shfl_xor_sync(0xffffffffu, e0, off));
  }
  if (lane != 0u) return;
  float4* rec = inst_wide + (size_t)i * kWideInstRows;
  rec[1].w = e1;
  rec[2].w = e0;
  // hits may lie before their box by the mesh's slack, its absolute part in world units along any direction
  const float stretch = sqrtf(dot(xyz(m.c0), xyz(m.c0)) + dot(xyz(m.c1), xyz(m.c1)) + dot(xyz(m.c2), xyz(m.c2)));
  // and by the margin: within twice its extent of the middle an absolute one, farther out a relative
  const float margin = fmaxf(4.0f * e1, 4.0f * (2.0f * extent * e1 + e0));
  const float slack = fminf(fmaxf(fmaxf(rec[4].z, rec[0].w * stretch), margin), kNoSlackBound);
  float l[3] = {b[0], b[1], b[2]}, u[3] = {b[3], b[4], b[5]};
  auto entry = [](const M4& x) {
    return fmaxf(fmaxf(max_abs3(xyz(x.c0)), max_abs3(xyz(x.c1))), max_abs3(xyz(x.c2)));
  };
  const float amp = entry(m) * entry(w);
  if (amp <= 8.0f) {
    const float tl[3] = {lo.x, lo.y, lo.z}, tu[3] = {hi.x, hi.y, hi.z};
    const float pad = 4e-6f * fmaxf(amp, 1.0f) * (fmaxf(max_abs3(lo), max_abs3(hi)) + max_abs3(sub(hi, lo)));
    for (int k = 0; k < 3; ++k) {
      const float x = fmaxf(l[k], tl[k] - pad), y = fminf(u[k], tu[k] + pad);
      if (x <= y) l[k] = x, u[k] = y;
    }
  }
  out[2 * (size_t)i] = make_float4(l[0], l[1], l[2], slack);
  const float ex = u[0] - l[0], ey = u[1] - l[1], ez = u[2] - l[2];
  out[2 * (size_t)i + 1] = make_float4(u[0], u[1], u[2], rec[5].w * (ex * ey + ey * ez + ez * ex));
}

__global__ void k_light_cdfs(const LightIn* __restrict__ lights, uint32_t n, const float4* __restrict__ prims,
                             float* tri_cdfs, float* mesh_areas) {
  const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n) return;
  const LightIn L = lights[l];
  float* cdf = tri_cdfs + L.cdf_offset;
  for (uint32_t t = 0; t < L.triangle_count; ++t) {
    const float4* p = prims + (size_t)(L.triangle_offset + t) * 3;
    const float3 p0 = xyz(p[0]), p1 = xyz(p[1]), p2 = xyz(p[2]);
    const float a = length(sub(p1, p0));
    const float b = length(sub(p2, p0));
    const float c = length(sub(p2, p1));
    const float s = 0.5f * (a + b + c);
    cdf[t] = sqrtf(s * (s - a) * (s - b) * (s - c));
  }
  float total = 0.0f;
  for (uint32_t t = 0; t < L.triangle_count; ++t) total = total + cdf[t];
  float prev = 0.0f;
  for (uint32_t t = 0; t < L.triangle_count; ++t) {
    const float cur = prev + cdf[t] / total;
    cdf[t] = cur;
    prev = cur;
  }
  mesh_areas[l] = total;
}

__global__ void k_strength_cdf(const LightIn* __restrict__ lights, uint32_t n, const float4* __restrict__ materials,
                               float* strength_cdf) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  float total = 0.0f;
  for (uint32_t l = 0; l < n; ++l) {
    const float3 em = xyz(materials[3 * (size_t)lights[l].material + 1]);
    const float s = dot(em, em);
    strength_cdf[l] = s;
    total = total + s;
  }
  float prev = 0.0f;
  for (uint32_t l = 0; l < n; ++l) {
    const float cur = prev + strength_cdf[l] / total;
    strength_cdf[l] = cur;
    prev = cur;
  }
}

}  // namespace

cudaError_t soup(const float* pos, const float* nrm, const float* uv, const uint32_t* idx, uint32_t ntris,
                 float4* prims, float4* tdata, cudaStream_t st) {
  if (!ntris) return cudaSuccess;
  k_soup<<<(ntris + 255) / 256, 256, 0, st>>>(pos, nrm, uv, idx, ntris, prims, tdata);
  return cudaGetLastError();
}

cudaError_t instances(const InstanceIn* in, uint32_t n, const float4* blas_nodes, float4* inst_out, float* bounds9,
                      float4* wide_out, cudaStream_t st, const uint32_t* slot) {
  if (!n) return cudaSuccess;
  k_instances<<<(n + 127) / 128, 128, 0, st>>>(in, n, blas_nodes, inst_out, bounds9, wide_out, slot);
  return cudaGetLastError();
}

cudaError_t tight_bounds(uint32_t n, const float4* instances, float4* inst_wide, const float* bounds9,
                         const float4* hulls, float4* out, cudaStream_t st) {
  if (!n) return cudaSuccess;
  k_tight_bounds<<<(n + 7) / 8, 256, 0, st>>>(n, instances, inst_wide, bounds9, hulls, out);
  return cudaGetLastError();
}

cudaError_t lights(const LightIn* lights, uint32_t n_lights, const float4* prims, const float4* materials,
                   float* tri_cdfs, float* mesh_areas, float* strength_cdf, cudaStream_t st) {
  if (!n_lights) return cudaSuccess;
  k_light_cdfs<<<(n_lights + 63) / 64, 64, 0, st>>>(lights, n_lights, prims, tri_cdfs, mesh_areas);
  k_strength_cdf<<<1, 32, 0, st>>>(lights, n_lights, materials, strength_cdf);
  return cudaGetLastError();
}

}  // namespace prep

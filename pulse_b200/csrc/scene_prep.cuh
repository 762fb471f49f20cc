// scene_prep.cuh -- device side of the reference's scene preparation systems.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace prep {

// prepare_extracted_mesh_assets (src/scene/mod.rs:410-424): triangle soup of
// positions and of normals/UVs through the index buffer (copies only).
cudaError_t soup(const float* pos, const float* nrm, const float* uv, const uint32_t* idx, uint32_t ntris,
                 float4* prims, float4* tdata, cudaStream_t st);

struct InstanceIn {
  float object_world[16];
  uint32_t triangle_offset, triangle_count, index_offset, node_offset, material_index;
  uint32_t wide_root, wide_leaf;  // root group of the mesh's eight-wide tree, or 0 and its only leaf
  float wide_slack, wide_slack_abs;
  uint32_t hull;            // the mesh's boxes for tight_bounds
  float wide_leaves;        // of a mesh without a slack: leaves that a line through it meets
  uint32_t pad;
};

// prepare_mesh_instances (src/scene/mod.rs:561-681) per instance: the 160 B
// record with the inverse transform, and the world bounds of the BLAS root
// (8 transformed corners) with their centre -> bounds9; the wide traversal's record
// (pt_wide.cuh) -> wide_out, unless it is null.  With `slot`, input i writes records and bounds slot[i] (an
// incremental update of some instances).
cudaError_t instances(const InstanceIn* in, uint32_t n, const float4* blas_nodes, float4* inst_out, float* bounds9,
                      float4* wide_out, cudaStream_t st, const uint32_t* slot = nullptr);

// Bounds (two float4) of each of the n instances for the wide traversal: around its
// mesh's 64 hull boxes transformed, instead of the corners of its root box; and in the first's w
// the instance's slack (pt_wide.cuh), relative and in world units, in the second's the area of its bounds
// times its mesh's wide_leaves.  Writes the distances' margins
// of its transform into its record.
cudaError_t tight_bounds(uint32_t n, const float4* instances, float4* inst_wide, const float* bounds9,
                         const float4* hulls, float4* out, cudaStream_t st);

struct LightIn { uint32_t instance, triangle_offset, triangle_count, cdf_offset, material; };

// create_triangle_area_cdf / create_emission_strength_cdf (src/scene/mod.rs:700-742),
// one thread per light (sequential sums in the reference's order).
cudaError_t lights(const LightIn* lights, uint32_t n_lights, const float4* prims, const float4* materials,
                   float* tri_cdfs, float* mesh_areas, float* strength_cdf, cudaStream_t st);

}  // namespace prep

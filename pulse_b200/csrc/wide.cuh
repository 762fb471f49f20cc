// wide.cuh -- the eight-wide trees of pt_wide.cuh, made from the binary ones.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace wide {

// Device words a collapse leaves for the host and the traversal.
enum Head : uint32_t {
  kRoot,    // a BLAS that is one leaf: its reference (pt_wide.cuh), else 0
  kCount,   // wide nodes
  kBad,     // nonzero: no wide tree (a box not finite or above 1e9, a leaf out of the references' range)
  kLevels,  // levels of the wide tree
  // How far the computed t of a hit may lie before its box (float bits): share of the
  // distance, and in units of the space.  A mesh's two (extents), or in the first the largest
  // of both of a TLAS's loose instances.
  kSlack, kSlackAbs,
  // Areas (floats): a mesh's leaf boxes (leaf_area), or a TLAS's instances without a bound times
  // their meshes' leaves; the root box.
  kAreas, kRootArea,
  kHeadWords = 8
};

// Most wide nodes a binary tree of n nodes can need (one per interior node).
constexpr uint32_t capacity(uint32_t n_nodes) { return (n_nodes + 1) / 2; }

// Collapses the tree of 32-byte nodes into out (capacity(n_nodes) x 96 bytes),
// with leaf_of[element slot] = index of the slot's leaf node.  queue: scratch of
// capacity(n_nodes) words.  Writes head's first four words.
cudaError_t collapse(const float4* nodes, uint32_t n_nodes, uint4* out, uint32_t* leaf_of, uint32_t* queue,
                     uint32_t* head, cudaStream_t st);

// The same for an instance tree, whose elements' leaf nodes go into the instances'
// records (pt_wide.cuh) and whose boxes are those of the instances' own bounds (two float4
// each, the first's w the instance's slack, the second's its share of kAreas; node_box: scratch of two float4 per node).  meta: the words of a
// bvh::build_direct queued before (kBad and nothing read if it failed), or nullptr.
cudaError_t collapse_tlas(const float4* nodes, uint32_t n_nodes, const uint32_t* meta, const uint32_t* instance_of,
                          float4* records, const float4* bounds, float4* node_box, uint4* out, uint32_t* queue,
                          uint32_t* head, cudaStream_t st);

// kHullBoxes boxes (two float4 each; unused ones inverted) that hold a mesh, from its
// collapsed tree (n_wide 0: its only node's box).
constexpr uint32_t kHullBoxes = 64;
cudaError_t hull(const uint4* wide_nodes, uint32_t n_wide, const float4* nodes, float4* out, cudaStream_t st);

// A mesh's n nodes with their indexes moved by node_add and their triangle slots by
// slot_add, as they go into the scene's array.
cudaError_t relocate(const uint32_t* nodes, uint32_t n, uint32_t node_add, uint32_t slot_add, uint32_t* out,
                     cudaStream_t st);

// Adds the areas of the leaf boxes of a tree of n_nodes nodes to head's kAreas, and its root's to
// kRootArea (zero to begin with).
cudaError_t leaf_area(const float4* nodes, uint32_t n_nodes, uint32_t* head, cudaStream_t st);

// Raises head's kSlack and kSlackAbs (zero to begin with) to those of n std430 triangles.
cudaError_t extents(const float4* prims, uint32_t n, uint32_t* head, cudaStream_t st);

}  // namespace wide

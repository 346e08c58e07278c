// Internal declarations shared by the host builder (nb_scene.cpp), the Sobol generator
// (nb_sobol.cpp) and the CUDA side (nb_api.cu / nb_kernels.cu).
//
// Device layout.  The reference uploads 32-byte BVH nodes, 160-byte instances, 48-byte
// vertices and a u32 index list, and its traversal loads both children of an inner node as
// two separate 32-byte nodes and every triangle through three indexed 48-byte vertex loads
// (raytracing_sw.wgsl:218-225, 275-279).  The device layout keeps the same trees but packs
// what one traversal step touches into 32-byte-aligned records read with 256-bit loads:
//   WideNode     96 B  8 children of a collapsed node: 8-bit quantised boxes
//   GpuTriPair   96 B  the one or two triangles of a leaf slot: v0, e1 = v1 - v0, e2 = v2 - v0 (the
//                      subtractions intersect_triangle performs) + the reference triangle indices
//   GpuInstTrace 64 B  the three rows of world_to_local used to transform rays, BLAS root,
//                      reference instance index
//   GpuInstShade 96 B  what intersect_scene/shading read from an instance
//   GpuVAttr     32 B  vertex normal + tangent (positions live in GpuTriPair)
// Triangles and instances are stored in the order of the wide trees' leaves.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/nbounce.h"

namespace nb {

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kLdsStride = 17u;      // pathtracing.wgsl:4 (fixed, independent of bounces)
constexpr uint32_t kLdsPerBounce = 2u;    // pathtracing.wgsl:2
constexpr uint32_t kMaxSampleCount = 1024u;  // pathtracer.rs:56

// The triangles of a leaf slot, one or two, component by component: [0] and [1] are the lanes of the
// packed triangle test.  A slot of one triangle has a degenerate second one (all zero: det = 0).
struct alignas(32) GpuTriPair {
  float v0[3][2], e1[3][2], e2[3][2];
  uint32_t ref_index[2];  // index in the reference's permuted triangle list (reported by hits)
  uint32_t pad[4];
};
struct alignas(32) GpuInstTrace {
  float row[3][4];     // row r = (W[0][r], W[1][r], W[2][r], W[3][r]) of world_to_local
  uint32_t blas_root;  // root of the instance's BLAS in the wide BLAS node array
  uint32_t ref_index;  // TLAS-permuted instance index of the reference (reported by hits)
  uint32_t pad[2];
};
struct alignas(16) GpuInstShade {
  float w2l_col[3][4];  // column c .xyz of world_to_local, .w = color[c]
  float l2w_row[3][4];  // row r .xyz of mat3(local_to_world), .w = roughness / metallic / emissive
};
struct alignas(16) GpuVAttr {
  float n[3];
  float tw;
  float t[3];
  float pad;
};
// 8-wide node collapsed from the reference's binary tree (96 B).  Child boxes are
// quantised to 8 bits per plane on a per-axis power-of-two grid anchored at p; the quantised
// boxes contain the exact ones.  Slot k is the inner child child_base + k or the leaf slot leaf_base + k
// (a GpuTriPair in a BLAS, a GpuInstTrace in the TLAS), by the mask of inner children and modulo 2^32;
// which order the slots have, and why: Collapser (nb_scene.cpp).  The masks and the grid steps lie ready
// for use, in words that the loads bring anyway, because the ALU pipe bounds the traversal: as counts and
// exponents to shift and mask, 1920x1080 at 64 spp took 94.0 instead of 92.6 ms, camera rays on the
// 1M-triangle soup 2.33 instead of 2.29.
struct alignas(32) WideNode {
  float p[3];
  uint32_t bits;       // children mask | inner children mask << 8 | grid step of z (float bits)
  uint32_t child_base;
  uint32_t leaf_base;
  float step[2];       // grid steps of x and y, powers of two
  uint8_t qlo_x[8], qlo_y[8], qlo_z[8], qhi_x[8], qhi_y[8], qhi_z[8];
  uint32_t pad[4];
  uint32_t n_children() const { return (uint32_t)__builtin_popcount(bits & 0xFFu); }
  uint32_t inner() const { return bits >> 8 & 0xFFu; }
  void set_children(uint32_t n, uint32_t inner) { bits |= ((1u << n) - 1u) | inner << 8; }
};
static_assert(sizeof(WideNode) == 96, "WideNode");
constexpr uint32_t kInstanceBit = 0x80000000u;  // TLAS stack entry that names an instance

static_assert(sizeof(GpuTriPair) == 96, "GpuTriPair");
static_assert(sizeof(GpuInstTrace) == 64, "GpuInstTrace");
static_assert(sizeof(GpuInstShade) == 96, "GpuInstShade");
static_assert(sizeof(GpuVAttr) == 32, "GpuVAttr");
static_assert(sizeof(nb_vertex) == 48 && sizeof(nb_bvh_node) == 32 && sizeof(nb_instance) == 160, "ref layout");

// Host copy of a scene: the reference-layout buffers and their device-layout translation.
struct HostScene {
  std::vector<nb_vertex> vertices;
  std::vector<uint32_t> indices;  // triangle-permuted (flatten_triangle_list)
  std::vector<nb_bvh_node> blas, tlas;
  std::vector<nb_instance> instances;  // TLAS-permuted

  std::vector<WideNode> wblas, wtlas;  // 8-wide trees; the TLAS root is wtlas[0]
  std::vector<uint32_t> wblas_root;    // per distinct BLAS root: index of its root in wblas
  size_t wblas_nodes = 0;  // size kept after the host copy is dropped
  size_t wtlas_nodes = 0;  // TLAS nodes without the gaps between them
  size_t tlas_entries = 0;                  // device TLAS leaves (itrace records without the gaps)
  bool has_tlas = false;
  std::vector<GpuInstTrace> itrace;
  std::vector<GpuInstShade> ishade;
  std::vector<GpuTriPair> tris;
  std::vector<GpuVAttr> vattr;
  double build_ms = 0.0;
};

// error reporting (thread-local message, nb_api.cu)
int fail(int status, const char* fmt, ...);

// nb_scene.cpp
int build_bvh_triangles(const float* positions, size_t n_vertices, const uint32_t* indices, size_t n_indices,
                        std::vector<nb_bvh_node>* nodes, std::vector<uint32_t>* permuted);
int build_scene_reference(const nb_vertex* vertices, size_t nv, const uint32_t* indices, size_t ni,
                          const nb_primitive* prims, size_t np, uint32_t flags, HostScene* out);
int adopt_reference_buffers(const nb_bvh_node* blas, size_t n_blas, const nb_bvh_node* tlas, size_t n_tlas,
                            const nb_instance* inst, size_t n_inst, const nb_vertex* v, size_t nv,
                            const uint32_t* idx, size_t ni, HostScene* out);
int to_device_layout(HostScene* s);

// nb_sobol.cpp
void sobol_burley_table(uint32_t n_samples, uint32_t n_dimsets, uint32_t seed, float* out);

}  // namespace nb

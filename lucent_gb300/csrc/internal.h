// Internal launcher declarations shared between the kernel files and the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../../include/lucent.h"
#include "api_util.h"
#include "common.cuh"

namespace lucent {

int grid_for(uint32_t n, int block);
int persistent_blocks(const void* kernel, int block);
void launch_pack_nodes(const float* ref_d, uint32_t count, Node* out_d, cudaStream_t s);
void launch_gather_tris(const float* pos_d, const uint32_t* idx_d, uint32_t tri_count, float4* out_d,
                        cudaStream_t s);
void launch_unpack(const Node* nodes, uint32_t count, const float4* tris, uint32_t tri_count, float* ref_d,
                   uint32_t* idx_d, cudaStream_t s);
// `ctr`: 8 zeroed words (error word, queue lengths, ray counters); `queue`: n words, 2 n with `near`.
struct NearTree;
void launch_closest(const Node* nodes, uint32_t node_count, const float4* tris, const float* rays_d, uint32_t n, double tMin,
                    double tMax, int32_t* prim, float* t, float* u, float* v, uint32_t* queue, uint32_t* ctr,
                    bool exact_only, bool top_levels, cudaStream_t s, const Node* wide = nullptr,
                    const NearTree* near = nullptr);
// Four-wide view of a binary node array (traverse_wide.cuh): 4 records per node.
void launch_wide_view(const Node* nodes, uint32_t node_count, Node* wide, cudaStream_t s);
// A few binary64 rays, a warp each (closest_hit.cu): rays in host memory (at
// most kPickArgs, passed by value) or on the device; results and error bits per ray.
constexpr uint32_t kPickArgs = 32;
struct PickHit {
  double t, u, v;
  int32_t prim;
  unsigned err;
};
void launch_pick(const Node* nodes, uint32_t node_count, const float4* tris, const double* rays, bool on_device,
                 uint32_t n, double tMin, double tMax, PickHit* out_d, cudaStream_t s);
void launch_closest_d(const Node* nodes, uint32_t node_count, const float4* tris, const double* rays_d, uint32_t n, double tMin,
                      double tMax, int32_t* prim, double* t, double* u, double* v, unsigned* err, cudaStream_t s);

// Nearest-first view of a tree (traverse_near.cuh, near_build.cu): records,
// each slot's leaf, the centre of the tree with the radius within which ray
// origins may lie, and how the box growth for farther origins rises with their
// distance. Not usable (and empty) for trees the argument does not
// cover, and where there is no memory for it. `tris`: slot order, 3 float4 each; lo, hi: the root's box.
struct NearTree {
  explicit NearTree(StreamUses* uses = nullptr) : records{nullptr, 0, uses}, leaf_of{nullptr, 0, uses} {}
  DeviceBuffer records, leaf_of;
  float4 bound = {0.f, 0.f, 0.f, 0.f};  // centre, radius
  float2 far = {0.f, 0.f};              // from this distance on, growth per unit of distance
  bool wide_range = false;              // the radius is 64 diagonals or more
  bool usable = false;
  void release() {
    records.release();
    leaf_of.release();
    usable = false;
  }
};
lucent_status build_near_view(const Node* nodes, uint32_t n_nodes, const float4* tris, uint32_t n_tris,
                              const float lo[3], const float hi[3], NearTree& out, cudaStream_t s);

// Texture arrays (texture.cu): decode tables (512: sRGB byte -> linear, then
// byte / 255) and sRGB code-value midpoints (255), the shared layer size
// (renderer.ts:316-322), and the resampling of each referenced image into its
// layer of a size x size RGBA8 array.
void texel_tables(float lut[512], float mid[255]);
int texture_array_size(const uint32_t* w, const uint32_t* h, const int32_t* layers, uint32_t n_layers);
lucent_status build_texture_layers(const uint8_t* const* images, const uint32_t* w, const uint32_t* h,
                                   const int32_t* layers, uint32_t n_layers, int size, bool srgb, const float* lut_d,
                                   const float* mid_d, uint8_t* out_d, cudaStream_t s);
// buildEnvSampler on the GPU (env_sampler.cu): the sampler grid of a w x h
// map, and the table (gw * gh float4) built from a device RGB map.
void env_grid(uint32_t w, uint32_t h, uint32_t max_w, uint32_t& gw, uint32_t& gh);
lucent_status gpu_env_sampler(const float* rgb_d, uint32_t w, uint32_t h, uint32_t max_w, uint32_t& gw, uint32_t& gh,
                              float4* table_d, double& total, cudaStream_t s);
// What a build returns: node count, depth and bounds always; the device layout
// (Node array, slot-order triangles, triIndices) and the reference's arrays on
// the host (8 floats a node, n indices) where given.
struct BuildOut {
  DeviceBuffer* nodes = nullptr;
  DeviceBuffer* tris = nullptr;
  DeviceBuffer* order = nullptr;
  float* nodes_host = nullptr;
  uint32_t* tri_host = nullptr;
  uint32_t node_count = 0, depth = 0;
  double bounds[6] = {0, 0, 0, 0, 0, 0};
};
lucent_status gpu_build_bvh(const float* pos_d, uint32_t n, int max_leaf, int bins, cudaStream_t s, BuildOut& out);

}  // namespace lucent

// Device builds of the two trees (gpu_bvh.cu, gpu_sah.cu) and of a scene's
// device arrays (gpu_scene.cu).
#pragma once
#include <cuda_runtime.h>

#include "bvh.h"

namespace cpppt_gb300 {

// Device allocations, freed with the list.
struct DeviceBufs {
    std::vector<void*> v;
    DeviceBufs() = default;
    DeviceBufs(const DeviceBufs&) = delete;
    DeviceBufs& operator=(const DeviceBufs&) = delete;
    ~DeviceBufs() { for (void* p : v) cudaFree(p); }
};

struct RefBuildStats {
    int levels = 0;  // tree levels (kernel launches of the level loop)
    int nodes = 0;   // internal nodes
};

// RefTopology in device memory.
struct RefTree {
    int32_t* leaf_order = nullptr;
    int32_t* rank = nullptr;
    int32_t* prim_parent = nullptr;
    int32_t* node_parent = nullptr;
    float4* node_box = nullptr;  // lower and upper corner of each node
    int n_nodes = 0;
};

// The same topology as build_ref_topology (bvh.cpp), bit for bit, built on
// the current device on stream st from tv (device, 9 floats per triangle).
// The boxes are allocated from `keep`, everything else from `scratch`.
// Synchronises st.  n_tris > 0.
RefTree build_ref_tree(const float* tv, int n_tris, cudaStream_t st, DeviceBufs& scratch, DeviceBufs& keep,
                       RefBuildStats* stats = nullptr);
// With input and results in host memory.
RefTopology build_ref_topology_device(const float* tri_v, int n_tris, cudaStream_t st, RefBuildStats* stats = nullptr);

struct WideBuildStats {
    int top_levels = 0;    // level-synchronous launches over nodes of more than 1024 triangles
    int subtrees = 0;      // CTAs that each split a subtree of at most 1024 triangles
    int binary_nodes = 0;  // nodes of the binary SAH tree
    int wide_levels = 0;   // breadth-first levels of the 4-wide tree
};

// WideBVH in device memory.
struct WideTree {
    uint4* nodes = nullptr;  // 4 per node
    int32_t* tri_order = nullptr;
    float* inflate = nullptr;
    int n_nodes = 0;
    int max_depth = 0;
};

// The same tree as build_wide_bvh (bvh.cpp), bit for bit (nodes, leaf order,
// depth, inflation), built on the current device on stream st (gpu_sah.cu)
// from tv as above.  The nodes are allocated from `keep`, everything else
// from `scratch`.  Synchronises st.  n_tris > 0.
WideTree build_wide_tree(const float* tv, int n_tris, int max_leaf, cudaStream_t st, DeviceBufs& scratch,
                         DeviceBufs& keep, WideBuildStats* stats = nullptr);
// With input and results in host memory.
WideBVH build_wide_bvh_device(const float* tri_v, int n_tris, int max_leaf, cudaStream_t st,
                              WideBuildStats* stats = nullptr);

// Scene arrays (gpu_scene.cu).  verts, nrms, tans (null: none): 3 floats per
// vertex; tri: 3 vertex indices per triangle, all in range.
// tv: 9 floats per triangle; vidx: {a, b, c, material}; key6 (zeroed): bounds
// keys for triangle_bounds.
void launch_triangle_positions(const float* verts, const int32_t* tri, const int32_t* material, int n, float* tv,
                               int4* vidx, uint32_t* key6, int num_sms, cudaStream_t st);
void launch_leaf_triangles(const float* tv, const int32_t* order, const int32_t* rank, const int32_t* parent, int n,
                           float4* tris, cudaStream_t st);
void launch_vertices(const float* verts, const float* nrms, const float* tans, int n, float4* vpos, float4* vnrm,
                     float4* vbt, cudaStream_t st);
// Bounds from host copies of the keys (infinite, lower above upper, without triangles).
void triangle_bounds(const uint32_t key6[6], float lo[3], float hi[3]);

}  // namespace cpppt_gb300

// bvh_build.hpp -- host binned-SAH BVH builder (deterministic output, parallel
// over subtrees) and its conversion to the GPU node layout.
//
// Same family as the reference builder (src/scene/bvhBuilder.cpp:115-312: binned
// SAH over centroids on all three axes, 16 bins, leaves of up to 4 triangles,
// median fallback) but written for this engine: bins are filled from per-triangle
// boxes computed once, the partition is by bin index so binning and splitting
// agree exactly, subtrees above a size threshold are built on separate threads,
// and the tree is renumbered in pre-order at the end so the node order does not
// depend on thread timing (the reference's atomic counter does,
// src/scene/bvhBuilder.cpp:245-248).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace sbr {

struct BuildOptions {
    int leaf_size = 4;     // split while more triangles than this
    int bin_count = 16;
    int n_threads = 0;     // 0 -> hardware concurrency
    int max_leaf = 15;     // hard cap (GPU leaf encoding)
};

struct BinNode {
    float lo[3], hi[3];
    int32_t left, right;   // child indices (-1 for leaves)
    int32_t first, count;  // triangle range in the permuted order (leaves)
};

struct BinTree {
    std::vector<BinNode> nodes;      // pre-order, root = 0
    std::vector<int32_t> order;      // slot -> caller triangle index
    int depth = 0;
};

// tri_lo/tri_hi: per-triangle boxes (3 floats each), used for the build.
BinTree build_sah(const std::vector<float>& tri_lo, const std::vector<float>& tri_hi, const BuildOptions& opt);

// The same tree built on the current CUDA device (gpu_build.cu) from the caller's
// vertices and triangles there: identical nodes, boxes and leaf triangle sets; triangles
// inside a leaf may be in another order.  Nodes are numbered breadth first.
struct GpuTree {
    int device = 0;
    char* block = nullptr;      // everything below, from the device's pool
    int n = 0, nnodes = 0, levels = 0;
    float* lo = nullptr;        // [nnodes * 3] boxes
    float* hi = nullptr;
    int32_t* left = nullptr;    // children, -1 for leaves
    int32_t* right = nullptr;
    int32_t* first = nullptr;   // triangle range of a leaf in `order`
    int32_t* count = nullptr;
    int32_t* order = nullptr;   // [n] slot -> caller triangle index
    // of the collapse: 4-wide nodes in breadth-first order, and where each level starts
    int ncollapsed = 0;
    int32_t* work = nullptr;
    int32_t* level_off = nullptr;   // a block of its own
};
cudaError_t gpu_tree_build(const float* d_xyz, const uint32_t* d_idx, int n, double scale, const BuildOptions& opt,
                           cudaStream_t stream, GpuTree& out);
// The tree on the host, in pre-order, as build_sah returns it.
cudaError_t gpu_tree_download(const GpuTree& t, cudaStream_t stream, BinTree& out);
// Collapses the tree to 4-wide nodes, choosing the same children in the same order as the
// host's collapse and numbering the nodes as it does.  The first call finds the nodes and
// their number, the second writes them, with the nodes of each depth (level_nodes, and
// their offsets on the host: level_off).
cudaError_t gpu_tree_collapse(GpuTree& t, int stack_depth, cudaStream_t stream);
cudaError_t gpu_tree_emit(const GpuTree& t, void* d_nodes, int32_t* d_level_nodes, std::vector<int32_t>& level_off,
                          cudaStream_t stream);
void gpu_tree_free(GpuTree& t, cudaStream_t stream);
// has_opposed_twins (tie_order.hpp) on the device: *d_flag becomes 1 when there are such.
// `table`: gpu_twins_table(n) words of scratch.
size_t gpu_twins_table(size_t n);
cudaError_t gpu_opposed_twins(const float* d_xyz, const uint32_t* d_idx, size_t n, int32_t* table, int32_t* d_flag,
                              cudaStream_t stream);

}  // namespace sbr

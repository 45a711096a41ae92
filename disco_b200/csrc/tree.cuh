// Far field by cells: the interface between the plan (capi.cu, field.cu,
// field_fp32.cu: tables) and the hierarchical sum (tree.cu).
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "field.cuh"

namespace disco {

// One piece of the table as the cell sum sees it: a ball that holds the
// piece's whole source (apex and vertices), and its records as byte offsets
// into the table.
struct alignas(16) TreePiece {
    double x, y, z, rho;
    uint32_t piece, rec;         // LinePiece and its first LineSeg
    int32_t terms;               // segments
    int32_t pad;
};
static_assert(sizeof(TreePiece) == 48, "tree piece layout");

// Appends the tree pieces of an FP64 line table after its bytes (sets aux_tree).
void append_tree_pieces(HostTable& T);

// The sum's shape for one atom count: chosen once per plan and count.
struct TreeShape {
    static constexpr int kMaxLevels = 18;
    bool use = false;
    int levels = 0;
    int m[kMaxLevels][3] = {};   // cells per axis
    int q[kMaxLevels] = {};      // nodes per axis of a cell
    double theta[kMaxLevels] = {};
    int split[kMaxLevels] = {};  // lanes that share a node's images
    int mf[3] = {}, qf = 0;      // the cells the atoms are sorted into
    int near_split = 1;          // lanes that share an atom's near images
    double cost = 0.0, direct = 0.0;
};

// Picks levels, orders and cells for n atoms by their operation counts;
// `use` is false where the plain sum over every image is cheaper.
TreeShape tree_shape(const HostTable& T, int64_t n, const double box[3], int images);

// Queues the sum on `stream`.  *ran is false (and nothing was queued) when the
// scratch memory could not be had: the caller then sums directly.
int launch_tree(const FieldArgs& a, const HostTable& T, const TreeShape& S, const double box[3], int sm_count,
                cudaStream_t stream, bool* ran, std::string& err);

// Scratch pool of the cell sum: one per device, shared by the plans that have
// used it and given back when the last of them goes.
void tree_pool_retain(int device);
void tree_pool_release(int device);

} // namespace disco

// Far field by cells: the interface between the plan (capi.cu, field.cu,
// field_fp32.cu: tables) and the hierarchical sum (tree.cu).
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "field.cuh"

namespace disco {

// Appends an FP64 table's tree pieces after its bytes (sets aux_tree); a line
// table's are made here, one per piece.
void append_tree_pieces(HostTable& T);

// The sum's shape for one atom count: chosen once per plan and count.
struct TreeShape {
    static constexpr int kMaxLevels = 24;
    bool use = false;
    int levels = 0;              // levels of cells with nodes
    int total = 0;               // and after them the levels of squares summed at the atoms
    int m[kMaxLevels][3] = {};   // cells per axis
    int q[kMaxLevels] = {};      // nodes per axis of a cell, equivalent loopons per axis of a square
    double theta[kMaxLevels] = {};
    double cut[kMaxLevels] = {}; // loopons: half edge of the largest square used as one source
    int np[kMaxLevels] = {};     // sources: tree pieces of that cut
    bool eq[kMaxLevels] = {};    // loopons: some of them summed through equivalent loopons
    int split[kMaxLevels] = {};  // lanes that share a node's images
    int mf[3] = {}, qf = 0;      // the cells the atoms are sorted into
    bool fine = false;           // the near pass goes by the final cells (else by the last level's)
    int near_split = 1;          // lanes that share an atom's near images
    double cost = 0.0, direct = 0.0;
};

// Picks levels, orders and cells for n atoms by their operation counts; `use`
// is false where the plain sum over every image is estimated to be faster.
TreeShape tree_shape(const HostTable& T, int64_t n, const double box[3], int images, int sm_count);

// Queues the sum on `stream`, *launches kernels.  None (nothing was queued) when
// the scratch memory could not be had: the caller then sums directly.
int launch_tree(const FieldArgs& a, const HostTable& T, const TreeShape& S, int sm_count,
                cudaStream_t stream, int* launches, std::string& err);

} // namespace disco

// pbt_batch_types.h -- descriptors shared by the batch host code
// (pbt_batch.cpp) and the persistent batch kernel (pbt_batch.cuh).
#pragma once

#include <cuda_runtime.h>

namespace pbt {

struct BatchTile {
    int m;
    int lanes;              // systems in the tile (<= 32)
    int rows;               // rows of the tile layout (largest N of its systems)
    int nseg;               // segments per system
    long long mat_off;      // doubles, in A/B/C and the factor workspace
    long long vec_off;      // doubles, in D
    long long red_mat_off;  // doubles, in the reduced A'/C' workspace
    long long red_vec_off;  // doubles, in the reduced d' workspace
};

struct BatchArgs {
    const double* a;
    const double* b;
    const double* c;
    double* d;
    double* aw;
    double* cw;
    double* ra;
    double* rc;
    double* rd;
    const BatchTile* tiles;
    const int* lane_rows;  // [tile*32 + lane]: N of that system, 0 for an empty lane
    const int2* items1;    // (tile, segment or -1 for a whole-line Thomas item)
    const int2* items3;    // (tile, segment)
    int n1, n3;
    int rows3;             // rows of the longest segment in items3
    int* head1;            // queue head, zeroed before every solve
    int* seg_done;         // per tile: segments done (zeroed before every solve)
    unsigned long long* status;  // zero pivots, range flag
    unsigned char* redo = nullptr;  // [tile*32 + lane]: lines that k_batch_cols left to k_batch_redo
};

// Packing between the caller's per-system layout and the tiled layout.
struct PackArgs {
    const BatchTile* tiles;
    const int* lane_rows;
    const int* sys_of;              // [tile*32 + lane]: system index, -1 = empty lane
    const long long* user_mat_off;  // per system
    const long long* user_vec_off;
    const int* chunk_start;         // per tile: prefix sum of its chunks of kPackRows rows
    int ntiles;
    int chunks;                     // of all tiles
};
constexpr int kPackRows = 64;

// Block sizes up to this may be solved by k_batch_cols (pbt_batch_cols.cu): a
// pair of warps per item (tile, group of systems) in items1, in CTAs of
// batch_cols_pairs consecutive items of one block size (group -1: none).
constexpr int kBatchColsMaxBlock = 6;
constexpr int kBatchColsMaxPairs = 4;
constexpr int batch_cols_pairs(bool ff) { return ff ? kBatchColsMaxPairs : 1; }
cudaError_t launch_batch_cols(const BatchArgs& ba, int ff, cudaStream_t s);
// Lines of several segments whose elimination from both ends met a zero pivot or
// grew, in their segments; after launch_batch_cols.
cudaError_t launch_batch_redo(const BatchArgs& ba, int ff, cudaStream_t s);

// The launches of block size M (pbt_batch.cuh; instantiated with the other
// kernels of (Num, M) in pbt_inst.cu).
template <class Num, int M>
cudaError_t launch_batch(const BatchArgs& ba, int warps, cudaStream_t s, int* grid_out);
cudaError_t launch_pack(const PackArgs& pa, const double* ua, const double* ub, const double* uc, const double* ud,
                        double* ta, double* tb, double* tc, double* td, double* ud_out, int dir, cudaStream_t s);

}  // namespace pbt

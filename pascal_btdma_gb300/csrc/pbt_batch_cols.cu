// pbt_batch_cols.cu -- an uneven batch in one launch, one lane per block column
// (pbt_cols.cuh), for the tiles of block sizes up to kBatchColsMaxBlock.
//
// Why: with one thread per system a tile's longest line is too long a chain of
// rows, so its lines are cut into segments, at 2.4 times block Thomas's
// arithmetic and a second pass over the factors; and a launch per block size
// leaves the GPU to its last few items four times a solve.  With one lane per
// column a row's chain is ~5 times shorter, and eliminated from both ends a
// line has half the rows, so that the longest lines finish within the time
// that the whole batch keeps the GPU busy: block Thomas's arithmetic, every
// value read once, all block sizes in one launch, longest items first.  The
// rule is cols_solve (pbt_batch.cpp).  Uneven batch of 32768 systems, N 16 ..
// 4096, m 2 .. 5, float-float (GB300): 13232 -> 10611 us a solve and unpack.
#include "pbt_batch_types.h"
#include "pbt_cols.cuh"

namespace pbt {

// A tile planned in one segment is solved from its first row on, each warp of
// the CTA a group of its own; one planned in several by both ends (twisted),
// the CTA's two warps on one group.
template <class Num, int M>
__device__ __forceinline__ void batch_cols(const BatchArgs& ba, const BatchTile& tl, int group, double* sh) {
    const int side = threadIdx.x >> 5;
    const bool twisted = tl.nseg > 1;
    const ColLane cl = col_lane<M>(tl.lanes, twisted ? group : 2 * group + side);
    const int rows = tl.rows, n0 = rows / 2, n = twisted ? (side ? rows - n0 : n0) : rows;
    const size_t plane = (size_t)32 * rows, at = (cl.live ? (size_t)cl.sys : 0) + (twisted && side ? (size_t)32 * (rows - 1) : 0);
    const size_t mo = (size_t)tl.mat_off + at, vo = (size_t)tl.vec_off + at;
    if (twisted)
        thomas_cols_body<Num, M, false, false, true>((side ? ba.c : ba.a) + mo, ba.b + mo, (side ? ba.a : ba.c) + mo,
                                                     ba.d + vo, ba.cw + mo, plane, side ? -32 : 32, n, true, ba.status,
                                                     cl, side, sh);
    else
        thomas_cols_body<Num, M, false>(ba.a + mo, ba.b + mo, ba.c + mo, ba.d + vo, ba.cw + mo, plane, 32, n, true,
                                        ba.status, cl);
}

template <class Num>
__global__ void __launch_bounds__(64, 8) k_batch_cols(const BatchArgs ba) {
    __shared__ double sh[2 * 32 * kBatchColsMaxBlock];
    const int2 it = ba.items1[blockIdx.x];
    const BatchTile tl = ba.tiles[it.x];
    switch (tl.m) {
        case 1: batch_cols<Num, 1>(ba, tl, it.y, sh); break;
        case 2: batch_cols<Num, 2>(ba, tl, it.y, sh); break;
        case 3: batch_cols<Num, 3>(ba, tl, it.y, sh); break;
        case 4: batch_cols<Num, 4>(ba, tl, it.y, sh); break;
        case 5: batch_cols<Num, 5>(ba, tl, it.y, sh); break;
        default: batch_cols<Num, 6>(ba, tl, it.y, sh); break;
    }
}
static_assert(kBatchColsMaxBlock == 6, "k_batch_cols lists block sizes 1..6");

cudaError_t launch_batch_cols(const BatchArgs& ba, int ff, cudaStream_t s) {
    if (ba.n1 <= 0) return cudaSuccess;
    if (ff)
        k_batch_cols<FF><<<(unsigned)ba.n1, 64, 0, s>>>(ba);
    else
        k_batch_cols<F64><<<(unsigned)ba.n1, 64, 0, s>>>(ba);
    return cudaGetLastError();
}

}  // namespace pbt

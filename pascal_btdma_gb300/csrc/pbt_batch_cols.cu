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
// 4096, m 2 .. 5 (GB300), us a solve and unpack: float-float segments 13232, this
// with one pair of warps a CTA 10710, two 9484, four 8891, eight 10178 -- with
// pairs of every block size on an SM, their unrolled rows miss the instruction
// cache (63 % hits, "no instruction" half of all stalls), with eight a CTA waits
// for its longest; FP64, whose rows are short, 23238, 23616, 25989, 35174.
#include "pbt_batch_types.h"
#include "pbt_cols.cuh"

namespace pbt {

// A tile planned in one segment is solved from its first row on, each warp of
// the pair a group of its own; one planned in several by both ends (twisted),
// the pair's two warps on one group.
template <class Num, int M>
__device__ __forceinline__ void batch_cols(const BatchArgs& ba, const BatchTile& tl, unsigned char* redo, int group,
                                           double* sh, int bar) {
    const int side = (threadIdx.x >> 5) & 1;
    const bool twisted = tl.nseg > 1;
    const ColLane cl = col_lane<M>(tl.lanes, twisted ? group : 2 * group + side);
    const int rows = tl.rows, n0 = rows / 2, n = twisted ? (side ? rows - n0 : n0) : rows;
    const size_t plane = (size_t)32 * rows, at = (cl.live ? (size_t)cl.sys : 0) + (twisted && side ? (size_t)32 * (rows - 1) : 0);
    const size_t mo = (size_t)tl.mat_off + at, vo = (size_t)tl.vec_off + at;
    if (twisted)  // guarded: y in the first planes of aw
        thomas_cols_body<Num, M, false, false, true>((side ? ba.c : ba.a) + mo, ba.b + mo, (side ? ba.a : ba.c) + mo,
                                                     ba.d + vo, ba.cw + mo, plane, side ? -32 : 32, n, true, ba.status,
                                                     cl, ba.aw + mo, redo + (cl.live ? cl.sys : 0), side, sh, bar);
    else
        thomas_cols_body<Num, M, false>(ba.a + mo, ba.b + mo, ba.c + mo, ba.d + vo, ba.cw + mo, plane, 32, n, true,
                                        ba.status, cl);
}

template <class Num>
__global__ void __launch_bounds__(64 * batch_cols_pairs(Num::kConv), 8 / batch_cols_pairs(Num::kConv))
    k_batch_cols(const BatchArgs ba) {
    constexpr int kPairs = Num::kConv ? kBatchColsMaxPairs : 1;  // batch_cols_pairs
    __shared__ double sh[kPairs][kTwistShared<kBatchColsMaxBlock>];
    const int pair = threadIdx.x >> 6;
    const int2 it = ba.items1[blockIdx.x * kPairs + pair];
    if (it.y < 0) return;  // the last CTA of a block size is not full
    const BatchTile tl = ba.tiles[it.x];
    unsigned char* const redo = ba.redo + (size_t)it.x * 32;
    switch (tl.m) {
        case 1: batch_cols<Num, 1>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
        case 2: batch_cols<Num, 2>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
        case 3: batch_cols<Num, 3>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
        case 4: batch_cols<Num, 4>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
        case 5: batch_cols<Num, 5>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
        default: batch_cols<Num, 6>(ba, tl, redo, it.y, sh[pair], 1 + pair); break;
    }
}

// The lines of several segments that k_batch_cols left (thomas_cols_body's Guard),
// in their segments, one CTA an item.  The guard and this launch cost the uneven
// batch above 8900 -> 9180 us (12 of it the launch).
template <class Num, int M>
__device__ __forceinline__ void batch_redo(const BatchArgs& ba, const BatchTile& tl, unsigned char* redo, int group) {
    redo_cols_group<Num, M, false>(ba.a + tl.mat_off, ba.b + tl.mat_off, ba.c + tl.mat_off, ba.d + tl.vec_off,
                                   ba.aw + tl.mat_off, ba.cw + tl.mat_off, ba.ra + tl.red_mat_off,
                                   ba.rc + tl.red_mat_off, ba.rd + tl.red_vec_off, 32, tl.lanes, tl.rows, tl.nseg, group,
                                   redo, false, ba.status);
}
template <class Num>
__global__ void __launch_bounds__(64, 4) k_batch_redo(const BatchArgs ba) {
    const int2 it = ba.items1[blockIdx.x];
    if (it.y < 0) return;
    const BatchTile tl = ba.tiles[it.x];
    if (tl.nseg <= 1) return;
    unsigned char* const redo = ba.redo + (size_t)it.x * 32;
    switch (tl.m) {
        case 1: batch_redo<Num, 1>(ba, tl, redo, it.y); break;
        case 2: batch_redo<Num, 2>(ba, tl, redo, it.y); break;
        case 3: batch_redo<Num, 3>(ba, tl, redo, it.y); break;
        case 4: batch_redo<Num, 4>(ba, tl, redo, it.y); break;
        case 5: batch_redo<Num, 5>(ba, tl, redo, it.y); break;
        default: batch_redo<Num, 6>(ba, tl, redo, it.y); break;
    }
}
static_assert(kBatchColsMaxBlock == 6, "k_batch_cols and k_batch_redo list block sizes 1..6");

cudaError_t launch_batch_cols(const BatchArgs& ba, int ff, cudaStream_t s) {
    if (ba.n1 <= 0) return cudaSuccess;
    const int pairs = batch_cols_pairs(ff != 0);
    if (ff)
        k_batch_cols<FF><<<(unsigned)(ba.n1 / pairs), 64 * pairs, 0, s>>>(ba);
    else
        k_batch_cols<F64><<<(unsigned)(ba.n1 / pairs), 64 * pairs, 0, s>>>(ba);
    return cudaGetLastError();
}
cudaError_t launch_batch_redo(const BatchArgs& ba, int ff, cudaStream_t s) {
    if (ba.n1 <= 0) return cudaSuccess;
    if (ff)
        k_batch_redo<FF><<<(unsigned)ba.n1, 64, 0, s>>>(ba);
    else
        k_batch_redo<F64><<<(unsigned)ba.n1, 64, 0, s>>>(ba);
    return cudaGetLastError();
}

}  // namespace pbt

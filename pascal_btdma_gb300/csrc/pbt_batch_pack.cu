// pbt_batch_pack.cu -- the batch's layout conversion between the caller's
// per-system arrays and the packed tiles (pbt_batch_pack / pbt_batch_unpack).
#include "pbt_batch_types.h"

namespace pbt {

// Packing between the caller's per-system layout (system s at its own
// offset, in the reference layout of a single system: X_s[row + N_s*e],
// e = i + m*j, D_s[row + N_s*i]) and the tiled layout.  `sys_of` maps a tile
// lane to its system (-1 = empty).  One CTA moves kPackRows rows of a tile,
// element plane by element plane: the per-system side is read (or written)
// along the rows, 512 bytes a system, the tiled side along the lanes, and the
// plane turns around in shared memory (odd stride).  One thread per (row,
// lane), which touched 32 separate 8-byte places a warp on the per-system
// side, took 6758 us to pack and 1284 to unpack the uneven
// batch of 32768 systems (24 M rows), against 2899 and 229.
__device__ __forceinline__ int find_tile(const int* chunk_start, int ntiles, int idx) {
    int lo = 0, hi = ntiles - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunk_start[mid] <= idx) lo = mid; else hi = mid - 1;
    }
    return lo;
}

constexpr int kPackThreads = 256;

// dir = 0: user -> tiled (A, B, C and D); dir = 1: tiled D -> user D.
__global__ void __launch_bounds__(kPackThreads) k_pack(const PackArgs pa, const double* ua, const double* ub,
                                                       const double* uc, const double* ud, double* ta, double* tb,
                                                       double* tc, double* td, double* ud_out, int dir) {
    __shared__ double plane[32][kPackRows + 1];
    __shared__ long long mat0[32], vec0[32];
    __shared__ int rows[32];  // of the lane's system; -1: empty lane
    constexpr int kPer = 32 * kPackRows / kPackThreads;
    const int t = find_tile(pa.chunk_start, pa.ntiles, (int)blockIdx.x);
    const BatchTile tl = pa.tiles[t];
    const int m = tl.m, mm = m * m, r0 = ((int)blockIdx.x - pa.chunk_start[t]) * kPackRows;
    if (threadIdx.x < 32) {
        const int s = pa.sys_of[t * 32 + threadIdx.x];
        rows[threadIdx.x] = s >= 0 ? pa.lane_rows[t * 32 + threadIdx.x] : -1;
        mat0[threadIdx.x] = s >= 0 ? pa.user_mat_off[s] : 0;
        vec0[threadIdx.x] = s >= 0 ? pa.user_vec_off[s] : 0;
    }
    __syncthreads();
    // Along the rows: row rr of lanes ll, ll + 4, ...; along the lanes: lane lx
    // of rows rx, rx + 8, ...
    const int rr = threadIdx.x % kPackRows, ll = threadIdx.x / kPackRows, lx = threadIdx.x % 32, rx = threadIdx.x / 32;
    constexpr int kLaneStep = kPackThreads / kPackRows, kRowStep = kPackThreads / 32;
    const int row = r0 + rr;
    if (dir == 0) {
        // A system shorter than its tile is padded to the tile's rows with
        // rows that decouple (A = C = 0, B = I, d = 0: x = 0 there), and its
        // last real row's C is zeroed (the non-cyclic solve treats it as zero):
        // every lane of a tile then has the tile's rows and the same segment
        // boundaries, so a warp's accesses stay coalesced.
        for (int p = 0; p < 3 * mm + m; ++p) {
            const int arr = p < 3 * mm ? p / mm : 3, e = p - arr * mm;  // A, B, C, D
            const double* src = arr == 0 ? ua : arr == 1 ? ub : arr == 2 ? uc : ud;
            double* dst = arr == 0 ? ta : arr == 1 ? tb : arr == 2 ? tc : td;
            double v[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int l = ll + j * kLaneStep, n = rows[l];
                const bool live = row < n - (arr == 2 ? 1 : 0);
                const double pad = (arr == 1 && n >= 0 && e % (m + 1) == 0) ? 1.0 : 0.0;
                v[j] = live ? __ldcs(src + (size_t)(arr == 3 ? vec0[l] : mat0[l]) + row + (size_t)n * e) : pad;
            }
            __syncthreads();  // the previous plane has been written
#pragma unroll
            for (int j = 0; j < kPer; ++j) plane[ll + j * kLaneStep][rr] = v[j];
            __syncthreads();
            const size_t d0 = (size_t)(arr == 3 ? tl.vec_off : tl.mat_off) + lx + (size_t)32 * tl.rows * e;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int r = r0 + rx + j * kRowStep;
                if (r < tl.rows) __stcs(dst + d0 + (size_t)32 * r, plane[lx][rx + j * kRowStep]);
            }
        }
    } else {
        for (int i = 0; i < m; ++i) {
            const size_t s0 = (size_t)tl.vec_off + lx + (size_t)32 * tl.rows * i;
            double v[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int r = r0 + rx + j * kRowStep;
                v[j] = r < tl.rows ? __ldcs(td + s0 + (size_t)32 * r) : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kPer; ++j) plane[lx][rx + j * kRowStep] = v[j];
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int l = ll + j * kLaneStep, n = rows[l];
                if (row < n) __stcs(ud_out + (size_t)vec0[l] + row + (size_t)n * i, plane[l][rr]);
            }
        }
    }
}

cudaError_t launch_pack(const PackArgs& pa, const double* ua, const double* ub, const double* uc, const double* ud,
                        double* ta, double* tb, double* tc, double* td, double* ud_out, int dir, cudaStream_t s) {
    if (pa.chunks <= 0) return cudaSuccess;
    k_pack<<<(unsigned)pa.chunks, kPackThreads, 0, s>>>(pa, ua, ub, uc, ud, ta, tb, tc, td, ud_out, dir);
    return cudaGetLastError();
}

}  // namespace pbt

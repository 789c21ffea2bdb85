// pbt_ring.cuh -- the single-segment block Thomas solve of batches that fill
// the GPU, its inputs brought by a producer warp through a ring that the whole
// CTA shares.
//
// Why: k_thomas waits for the loads of a row where the row begins, FP64 with
// every warp of its own, float-float with the whole CTA, whose warps run the
// same rows together.  k_thomas_staged hides the loads, but its one-warp CTAs
// drift apart and each runs a ring of its own.  Here W consumer
// warps (one system a lane) take block columns, M values of every system, in
// the order the row uses them, from one ring of R slots; warp W issues them as
// bulk tensor copies (cp.async.bulk.tensor, one box of 32 systems x M planes a
// consumer warp) and is the only one to wait for free slots.  No consumer
// computes an address or holds a prefetched column, and no warp can run more
// than R columns ahead of another, which keeps them in step without a barrier.
//
// Measured (GB300, us, k_thomas -> this kernel): FP64 m = 5 65536 x 256 12665
// -> 12204 (its pipe is the bound: 10.7 ms of it), m = 6 x 128 10368 -> 9988,
// 100000 x 64 m = 4 2946 -> 2657, m = 6 8503 -> 7529; float-float m = 4
// 65536 x 256 3524 -> 3038, m = 3 1996 -> 1917, 100000 x 64 878 -> 667.  Not
// float-float m = 5, 6 (4890 -> 5170, 4515 -> 5100): bound by issue there, and
// the waits and releases of 22 items a row are 14 % more instructions.
//
// Items.  Forward, row q: d_q, the columns of B_q, of A_q, of C_q (A_0 and
// C_{N-1} come along unused, so that every row has 1 + 3M).  Backward, row q =
// N-2 .. 0: y_q, the columns of C'_q.  The arithmetic and its order are
// thomas_body_lu's, so the bits are k_thomas's.
//
// Protocol.  full[s]: one arrival (the producer's expect_tx) and the bytes;
// empty[s]: one arrival a consumer warp, after its lanes have read the slot.
// Between the sweeps every lane fences its generic stores (C', y) against the
// async proxy and the warps arrive at `turn`, which the producer waits for.
// Every wait is bounded (mbar_wait); when one runs out, the warp marks the
// status word and leaves, the others' waits run out in turn, and the producer
// waits (bounded) for the copies in flight before it ends.
//
// Lines by strides: dimensions {lines along the fast index, rows, outer lines,
// planes}, the two middle ones in the order of their strides (row_first).  A
// consumer warp's 32 lines lie along the fast index: lin % 32 == 0, or one run.
#pragma once

#include "pbt_staged.cuh"

namespace pbt {

__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap* map, int x, int y, int z, int w,
                                            unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_load_5d(unsigned dst, const CUtensorMap* map, int x, int y, int z, int w, int v,
                                            unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(v), "r"(bar)
        : "memory");
}

constexpr int kRingSlots = 8;  // at most

__device__ __forceinline__ unsigned global_ns_low() {
    unsigned t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}
// Waits for the phase, at most 2 s, or until some warp of the CTA has given up
// (`failed`, in shared memory).  Inline: a call would save the caller's
// registers to local memory around every wait that does not pass at once.
__device__ __forceinline__ void ring_wait(unsigned bar, unsigned parity, volatile int* failed) {
    if (mbar_try_wait(bar, parity)) return;
    const unsigned t0 = global_ns_low();
    while (!mbar_try_wait(bar, parity)) {
        if (*failed || global_ns_low() - t0 > (unsigned)kWaitLimitNs) {
            *failed = 1;
            break;
        }
    }
}

// The producer warp: every item of both sweeps, in order.  Transposed (the
// adjoint): A_q, B_q, C_q are C_{q-1}^T, B_q^T, A_{q+1}^T of the blocks as they
// are stored; their maps split the planes into the block's two indices, so
// that a column is a box along the second one, and the rows q - 1 and q + 1
// past either end come as zeros.
template <int M, bool Transposed>
__device__ __forceinline__ void ring_produce(const ThomasMaps& maps, const SolveArgs& g, const LineStrides& ls,
                                             int row_first, int warps, int active, int slots, unsigned ring_s,
                                             unsigned full_s, unsigned empty_s, unsigned turn_s,
                                             volatile int* failed) {
    const int lane = threadIdx.x & 31, N = g.nrow;
    const int s0 = (blockIdx.x * warps + lane) * 32;  // first system of consumer warp `lane`
    const int x = s0 % ls.lin, outer = s0 / ls.lin;
    const unsigned item_bytes = M * 256u, slot_bytes = item_bytes * warps;
    int slot = 0, issued = 0;
    unsigned phase = 1;  // parity of empty[slot] to wait for: a fresh barrier passes parity 1
    bool ok = true;
    auto issue = [&](const CUtensorMap* map, int row, int j, bool block) {
        ring_wait(empty_s + 8u * slot, phase, failed);
        ok = __all_sync(0xffffffffu, !*failed);
        if (!ok) return;
        fence_proxy_async_shared();
        if (lane == 0) mbar_expect_tx(full_s + 8u * slot, item_bytes * active);
        __syncwarp();
        if (lane < active) {
            const unsigned dst = ring_s + slot_bytes * slot + item_bytes * lane;
            const int y = row_first ? row : outer, z = row_first ? outer : row;
            if (Transposed && block)
                tma_load_5d(dst, map, x, y, z, j, 0, full_s + 8u * slot);
            else
                tma_load_4d(dst, map, x, y, z, j * M, full_s + 8u * slot);
        }
        ++issued;
        if (++slot == slots) {
            slot = 0;
            phase ^= 1u;
        }
    };
    for (int q = 0; q < N && ok; ++q) {
        issue(&maps.d, q, 0, false);
        for (int j = 0; j < M && ok; ++j) issue(&maps.b, q, j, true);
        for (int j = 0; j < M && ok; ++j) issue(&maps.a, Transposed ? q - 1 : q, j, true);
        for (int j = 0; j < M && ok; ++j) issue(&maps.c, Transposed ? q + 1 : q, j, true);
    }
    if (ok) {
        ring_wait(turn_s, 0, failed);
        ok = __all_sync(0xffffffffu, !*failed);
    }
    for (int q = N - 2; q >= 0 && ok; --q) {
        issue(&maps.d, q, 0, false);
        for (int j = 0; j < M && ok; ++j) issue(&maps.w, q, j, false);
    }
    // No copy may land after the CTA has ended: wait (bounded) for the last ones.
    if (lane == 0) {
        for (int n = issued > slots ? issued - slots : 0; n < issued; ++n) {
            const unsigned bar = full_s + 8u * (n % slots), par = (unsigned)(n / slots) & 1u;
            if (!mbar_try_wait(bar, par)) mbar_wait_slow(bar, par, kWaitLimitNs / 4);
        }
    }
    __syncwarp();
}

// The consumers also meet at the top of every row where the code of a row is
// long (float-float m = 4, 65536 x 256: 3124 -> 3038 us); the ring alone keeps
// the shorter ones close enough (m = 3 1917 us either way, FP64 m = 5 12204
// and 12211).
template <class Num, int M>
__host__ __device__ constexpr bool ring_step() {
    return Num::kConv && M >= 4;
}

// Guard: as thomas_cols_body (pbt_cols.cuh), but y stays in D and d is kept in
// g.aw's first planes (`saved` of k_redo_cols): 16384 x 512, FP64 m = 4, 5590 us
// unguarded, 5660 so, 5750 with y there.
template <class Num, int M, bool Transposed, bool Guard>
__global__ void __launch_bounds__(256, 2) k_thomas_ring(const __grid_constant__ ThomasMaps maps, const SolveArgs g,
                                                        const LineStrides ls, int row_first, int slots,
                                                        unsigned char* redo) {
    using T = typename Num::T;
    using Acc = typename Num::Acc;
    extern __shared__ __align__(128) double ring[];  // slots x warps x M x 32, then C'_{q-1} and y_{q-1}
    __shared__ __align__(8) unsigned long long bars[2 * kRingSlots + 1];
    __shared__ int failed;
    const int warps = (int)(blockDim.x >> 5) - 1, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.x * warps;  // of the batch's warps of 32 systems
    const int active = min(warps, (g.nsys + 31) / 32 - first);
    const unsigned full_s = smem_u32(bars), empty_s = full_s + 8u * kRingSlots, turn_s = full_s + 16u * kRingSlots;
    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(full_s + 8u * s, 1);
            mbar_init(empty_s + 8u * s, active);
        }
        mbar_init(turn_s, active);
        failed = 0;
        fence_mbar_init();
    }
    __syncthreads();
    if (w == warps) {
        ring_produce<M, Transposed>(maps, g, ls, row_first, warps, active, slots, smem_u32(ring), full_s, empty_s, turn_s,
                        &failed);
        return;
    }
    if (w >= active) return;

    const int N = g.nrow, sys = (first + w) * 32 + lane;
    const bool live = sys < g.nsys, raw = g.factors_raw != 0;
    const int cstride = warps * 32;
    double* const cps = ring + (size_t)slots * warps * M * 32 + w * 32 + lane;
    const size_t o0 = live ? (size_t)(sys % ls.lin) * (size_t)ls.in + (size_t)(sys / ls.lin) * (size_t)ls.out : 0;
    double* const D = g.d + o0;
    double* const CW = g.cw + o0;
    const size_t plane0 = (size_t)ls.elem, rs = (size_t)ls.row;
    const double* const sp0 = ring + w * (M * 32) + lane;
    const double* sp = sp0;
    int slot = 0;
    unsigned phase = 0;
    // The next item's column into v (value i of this lane's system in v[i]).
    auto take = [&](double (&v)[M]) {
        ring_wait(full_s + 8u * slot, phase, &failed);
#pragma unroll
        for (int i = 0; i < M; ++i) v[i] = sp[32 * i];
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_s + 8u * slot);
        sp += (size_t)cstride * M;
        if (++slot == slots) {
            slot = 0;
            sp = sp0;
            phase ^= 1u;
        }
    };
    unsigned bad = 0, amax = 0;
    [[maybe_unused]] float size = 0.f;  // of C'
    for (int q = 0; q < N; ++q) {
        if constexpr (ring_step<Num, M>()) asm volatile("barrier.sync 1, %0;" ::"r"(active * 32) : "memory");
        const size_t o = (size_t)q * rs;
        const bool last = q == N - 1;
        Acc r[M][M], xd[M];
        {
            double v[M];
            take(v);
#pragma unroll
            for (int i = 0; i < M; ++i) xd[i] = Num::acc(Num::in_rhs(&v[i]));
            if constexpr (Guard) {
                if (live) {
#pragma unroll
                    for (int i = 0; i < M; ++i) __stcs(g.aw + o0 + o + (size_t)i * plane0, v[i]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < M; ++j) {
            double v[M];
            take(v);
#pragma unroll
            for (int i = 0; i < M; ++i) r[i][j] = Num::acc(Num::in(&v[i]));
        }
#pragma unroll 1
        for (int k = 0; k < M; ++k) {
            double v[M];
            take(v);
            if (q > 0) {
                T ck[M];
#pragma unroll
                for (int j = 0; j < M; ++j) ck[j] = Num::lds(cps + (k * M + j) * cstride);
                const T yk = Num::lds(cps + (M * M + k) * cstride);
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    const T a = Num::in(&v[i]);
#pragma unroll
                    for (int j = 0; j < M; ++j) Num::msub(r[i][j], a, ck[j]);
                    Num::msub(xd[i], a, yk);
                }
            }
        }
        LU<Num, M> lu;
        lu_factor<Num, M>(r, lu, bad);
        const size_t plane = opaque(plane0);
        double* pw = CW + o;
        // y as column -1 of the column loop: one copy of the solve's code.
#pragma unroll 1
        for (int j = -1; j < M; ++j) {
            Acc cj[M];
            T xj[M];
            if (j < 0) {
#pragma unroll
                for (int i = 0; i < M; ++i) cj[i] = xd[i];
            } else {
                double v[M];
                take(v);
                if (last) continue;
#pragma unroll
                for (int i = 0; i < M; ++i) cj[i] = Num::acc(Num::in(&v[i]));
            }
            lu_solve<Num, M>(lu, cj, xj);
            if (j < 0) {
#pragma unroll
                for (int i = 0; i < M; ++i) Num::sts(cps + (M * M + i) * cstride, xj[i]);
                if (live) {
                    if (last)
                        out_vec<Num, M>(D + o, plane, xj, amax);
                    else
                        st_raw_vec<Num, M>(D + o, plane, xj);
                }
            } else {
#pragma unroll
                for (int i = 0; i < M; ++i, pw += plane) {
                    if constexpr (Guard) size = max_nan(size, Num::size(xj[i]));
                    if (live) {
                        if (raw || !Num::kConv)
                            Num::sts(pw, xj[i]);
                        else
                            Num::out(pw, xj[i]);
                    }
                    Num::sts(cps + (i * M + j) * cstride, xj[i]);
                }
            }
        }
    }
    {
        T y[M];
#pragma unroll
        for (int i = 0; i < M; ++i) y[i] = Num::lds(cps + (M * M + i) * cstride);
        // The backward sweep reads what this warp stored through the async proxy.
        fence_proxy_async_global();
        __syncwarp();
        if (lane == 0) mbar_arrive(turn_s);
        for (int q = N - 2; q >= 0; --q) {
            const size_t o = (size_t)q * rs;
            double v[M];
            take(v);
            Acc s[M];
#pragma unroll
            for (int i = 0; i < M; ++i) s[i] = Num::acc(Num::from_raw(v[i]));
#pragma unroll
            for (int k = 0; k < M; ++k) {
                take(v);
#pragma unroll
                for (int i = 0; i < M; ++i) Num::msub(s[i], ld_fac<Num>(&v[i], raw), y[k]);
            }
#pragma unroll
            for (int i = 0; i < M; ++i) y[i] = Num::fin(s[i]);
            if (live) out_vec<Num, M>(D + o, opaque(plane0), y, amax);
        }
    }
    __syncwarp();
    if (*(volatile int*)&failed) {
        if (lane == 0) atomicAdd(g.status, kStallMark);
        return;
    }
    if constexpr (Guard) {
        if (live && (bad != 0 || Num::grown(size))) {
            redo[sys] = 1;
            return;
        }
    }
    if (live) report_status(g.status, bad | range_bits<Num>(amax, true));
}

// Consumer threads a CTA: as in_step_tpb, at most 224 (with the producer, two
// CTAs of 256 threads of 128 registers an SM), so that the CTAs make whole
// waves; as many ring slots as two CTAs an SM leave shared memory for.
template <class Num, int M, bool Transposed, bool Guard>
cudaError_t launch_ring(const SolveArgs& g, const LineStrides& ls, const ThomasMaps& maps, int row_first,
                        unsigned char* redo) {
    const auto kernel = k_thomas_ring<Num, M, Transposed, Guard>;
    const long long sms = g.sms > 0 ? g.sms : 1, cap = 224;
    const long long waves = (g.nsys + cap * sms - 1) / (cap * sms);
    const int warps = (int)((((long long)g.nsys + waves * sms - 1) / (waves * sms) + 31) / 32);
    const size_t slot = (size_t)warps * M * 256, fixed = (size_t)warps * (M * M + M) * 256;
    const size_t budget = 113u * 1024u;
    if (warps < 1 || warps > 7 || fixed + 2 * slot > budget) return cudaErrorNotSupported;
    size_t slots = (budget - fixed) / slot;
    if (slots > kRingSlots) slots = kRingSlots;
    const size_t smem = fixed + slots * slot;
    if (const cudaError_t e = allow_smem(kernel, smem); e != cudaSuccess) return e;
    const unsigned grid = (unsigned)(((g.nsys + 31) / 32 + warps - 1) / warps);
    kernel<<<grid, 32 * (warps + 1), smem, g.stream>>>(maps, g, ls, row_first, (int)slots, redo);
    return cudaGetLastError();
}
// Guarded plans take the ring in FP64 from m = 4 on only.
template <class Num, int M, bool Transposed>
cudaError_t launch_ring(const SolveArgs& g, const LineStrides& ls, const ThomasMaps& maps, int row_first,
                        unsigned char* redo) {
    if (redo == nullptr) return launch_ring<Num, M, Transposed, false>(g, ls, maps, row_first, redo);
    if constexpr (!Num::kConv && M >= 4) return launch_ring<Num, M, Transposed, true>(g, ls, maps, row_first, redo);
    return cudaErrorNotSupported;
}
template <class Num, int M>
cudaError_t launch_thomas_ring(const SolveArgs& g, const LineStrides& ls, const ThomasMaps& maps, int row_first,
                               unsigned char* redo) {
    return launch_ring<Num, M, false>(g, ls, maps, row_first, redo);
}
template <class Num, int M>
cudaError_t launch_transposed_ring(const SolveArgs& g, const LineStrides& ls, const ThomasMaps& maps,
                                   unsigned char* redo) {
    return launch_ring<Num, M, true>(g, ls, maps, 1, redo);
}

}  // namespace pbt

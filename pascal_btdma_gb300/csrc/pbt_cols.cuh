// pbt_cols.cuh -- the solver with one lane per block column, for batches that
// one thread per system (or per segment) leaves the GPU nearly idle with.
//
// Why: a thread that carries a whole block row runs ~2.3 m^3 multiply-adds a
// row one after another, so a batch of a few thousand systems has one warp an
// SM or less, each stepping through its rows at the latency of that chain
// (FP64, m = 3: 4.8 us a row, 1024 systems).  Here a group of m + 1 lanes
// carries a system: lane j < m holds column j of R_q, of C'_q (and of A'_q in
// the local stage), lane m the right-hand side, which takes the place of a
// column in every phase, so no lane branches:
//   [R | t] = [B | d] - A [C' | y]   column by column, A's columns broadcast by
//                                    shuffles (a_ik from lane k);
//   elimination of R                 lane k finds the pivot of step k and the
//                                    multipliers, which go to the group;
//   [C' | y] = R^{-1} [C | t]        every lane its own column.
// A warp holds 32 / (m + 1) systems; the chain of a row falls from ~2.3 m^3 to
// ~2.5 m^2 dependent steps, and a batch has m + 1 times the threads.  The price
// is work in idle slots (the reciprocals, lane m beside R), 1.7 times the
// multiply-adds at m = 5: where one thread per system fills the GPU that is the
// better form (the rule and its figures: cols_pay, pbt_api.cpp).
// A lane's inputs of the next row are loaded while this row is eliminated.
// Every element sees the operations of thomas_body / modi_body / reduced_body
// (gesv) in the same order, so the bits are theirs.
#pragma once

#include "pbt_kernels.cuh"

namespace pbt {

template <int M>
__host__ __device__ constexpr int cols_systems() {
    return 32 / (M + 1);  // systems per warp
}

__device__ __forceinline__ double col_bcast(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ ff col_bcast(ff v, int src) {
    return {__shfl_sync(0xffffffffu, v.h, src), __shfl_sync(0xffffffffu, v.l, src)};
}

// This lane's place: group of system `sys`, column j (m: the right-hand side),
// `base` the group's first lane.  Lanes past the last group and groups past the
// last system are not live: they run along on zeros and store nothing.
struct ColLane {
    int j, base;
    long long sys;
    bool live;
};
template <int M>
__device__ __forceinline__ ColLane col_lane(long long nsys, long long warp) {
    constexpr int G = M + 1, S = cols_systems<M>();
    const int lane = threadIdx.x & 31;
    ColLane c;
    const bool idle = lane >= S * G;
    const int g = idle ? S - 1 : lane / G;
    c.j = idle ? M : lane - g * G;
    c.base = g * G;
    c.sys = warp * S + g;
    c.live = !idle && c.sys < nsys;
    return c;
}
// This warp's number in the grid.
__device__ __forceinline__ long long grid_warp() {
    return (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}

// Barrier `id` of the 64 threads of a pair of warps.
__device__ __forceinline__ void pair_barrier(int id) { asm volatile("barrier.sync %0, 64;" ::"r"(id) : "memory"); }

// M values `stride` apart at p (zeros on a lane that is not live), raw.
template <int M>
__device__ __forceinline__ void col_load(double (&v)[M], const double* p, size_t stride, bool live) {
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = live ? p[(size_t)i * stride] : 0.0;
}

// One elimination of the group's R (lane j < M: column j in r; consumed) on NX
// right-hand sides a lane (x), solutions in x.  gesv, column per lane.
template <class Num, int M, int NX>
__device__ __forceinline__ void col_gesv(typename Num::Acc (&r)[M], typename Num::Acc (&x)[NX][M], const ColLane& cl,
                                         unsigned& bad) {
    using T = typename Num::T;
    using Acc = typename Num::Acc;
    T u[M];     // this column of U (rows 0..j), normalised
    T rinv[M];  // the group's 1 / U_kk
    steps_up<0, M>([&](auto kc) {
        const int k = kc;
        const int src = cl.base + k;
        if (k + 1 < M) {
            int p = k;
            auto best = Num::akey(r[k]);
#pragma unroll
            for (int i = k + 1; i < M; ++i) {
                const auto v = Num::akey(r[i]);
                const bool gt = v > best;
                best = gt ? v : best;
                p = gt ? i : p;
            }
            p = __shfl_sync(0xffffffffu, p, src);
            if (__any_sync(0xffffffffu, p != k)) {
#pragma unroll
                for (int i = k + 1; i < M; ++i) {
                    const unsigned s = (p == i);
                    const Acc t = r[k];
                    r[k] = Num::asel(s, r[i], t);
                    r[i] = Num::asel(s, t, r[i]);
#pragma unroll
                    for (int h = 0; h < NX; ++h) {
                        const Acc y = x[h][k];
                        x[h][k] = Num::asel(s, x[h][i], y);
                        x[h][i] = Num::asel(s, y, x[h][i]);
                    }
                }
            }
        }
        u[k] = Num::fin(r[k]);
        const bool mine = cl.j == k;
        if (mine) bad |= Num::is_zero(u[k]);
        // Only lane k's reciprocal is used; the others take that of 1, so that
        // their zeros and subnormals do not send the warp the slow way.
        const T ri = Num::rcp(Num::sel(mine, u[k], Num::one()));
        rinv[k] = col_bcast(ri, src);
        T xk[NX];
#pragma unroll
        for (int h = 0; h < NX; ++h) {
            xk[h] = Num::fin(x[h][k]);
            x[h][k] = Num::acc(xk[h]);
        }
#pragma unroll
        for (int i = k + 1; i < M; ++i) {
            const T l = col_bcast(Num::mul(Num::fin(r[i]), ri), src);
            Num::msub(r[i], l, u[k]);
#pragma unroll
            for (int h = 0; h < NX; ++h) Num::msub(x[h][i], l, xk[h]);
        }
    });
    steps_down<M - 1, M>([&](auto kc) {
        const int k = kc;
        T xk[NX];
#pragma unroll
        for (int h = 0; h < NX; ++h) {
            xk[h] = Num::mul(Num::fin(x[h][k]), rinv[k]);
            x[h][k] = Num::acc(xk[h]);
        }
#pragma unroll
        for (int i = 0; i < k; ++i) {
            const T uk = col_bcast(u[i], cl.base + k);
#pragma unroll
            for (int h = 0; h < NX; ++h) Num::msub(x[h][i], uk, xk[h]);
        }
    });
}

// acc[i] -= sum over k of (column k's v[i]) * c[k], k ascending: a product with
// a block whose column k is in lane k.
template <class Num, int M>
__device__ __forceinline__ void col_product(typename Num::Acc (&acc)[M], const typename Num::T (&v)[M],
                                            const typename Num::T (&c)[M], int base) {
#pragma unroll
    for (int k = 0; k < M; ++k)
#pragma unroll
        for (int i = 0; i < M; ++i) Num::msub(acc[i], col_bcast(v[i], base + k), c[k]);
}
// Two products with the same block.
template <class Num, int M>
__device__ __forceinline__ void col_product2(typename Num::Acc (&acc)[M], typename Num::Acc (&acd)[M],
                                             const typename Num::T (&v)[M], const typename Num::T (&c)[M],
                                             const typename Num::T (&d)[M], int base) {
#pragma unroll
    for (int k = 0; k < M; ++k)
#pragma unroll
        for (int i = 0; i < M; ++i) {
            const typename Num::T a = col_bcast(v[i], base + k);
            Num::msub(acc[i], a, c[k]);
            Num::msub(acd[i], a, d[k]);
        }
}

// The outcome of a lane's group: its pivots and the largest value it wrote.
template <int M>
__device__ __forceinline__ void col_merge(unsigned& bad, unsigned& amax, const ColLane& cl) {
    unsigned b = 0, a = 0;
#pragma unroll
    for (int k = 0; k <= M; ++k) {
        b |= __shfl_sync(0xffffffffu, bad, cl.base + k);
        a = max(a, __shfl_sync(0xffffffffu, amax, cl.base + k));
    }
    bad = b;
    amax = a;
}
// Reported once a system, with the range check of the values it wrote.
template <class Num, int M>
__device__ __forceinline__ void col_report(unsigned long long* status, unsigned bad, unsigned amax, bool whole,
                                           const ColLane& cl) {
    col_merge<M>(bad, amax, cl);
    if (cl.live && cl.j == 0) report_status(status, bad | range_bits<Num>(amax, whole));
}

// Rows of C' and y that the backward sweep has in flight.
template <int M>
__host__ __device__ constexpr int cols_ahead() {
    return M <= 5 ? 4 : 2;
}

// Single-segment block Thomas of one system per group.  Pointers at the
// system's first row; Reduced: the reduced system of the two-stage method (B =
// I, everything raw; A, C', d in RA, RC, RD); Transposed: A, B and C hold the
// transposed blocks (column j of a block is row j of what is stored).
//
// Guard: for lines that the plan cuts into segments, whose two-stage method
// needs other blocks to be regular than an elimination from the ends does (the
// last block, singular in a line closed by a constraint, is one that it never
// inverts).  The forward sweep leaves y in Y instead of D and follows the size
// of C' (kGrowthExp).  A line that met a zero pivot or grew past it keeps d, its
// flag *redo is set, and k_redo_cols solves it in its segments; otherwise D takes
// x.  Unguarded -> guarded, us, where nothing is redone: FP64 m = 3, 1024 x 128
// 151.5 -> 153.6 (2 of it k_redo_cols' launch), float-float m = 3, 12347 x 301
// 642 -> 663, FP64 m = 8, 4096 x 1024 24886 -> 25012; where every line is:
// FP64 m = 5, 1000 x 128 in 4 432 -> 986 (the two-stage method alone, one thread a
// segment, 1569).
//
// Twisted: the line is eliminated from both ends at once, by two warps of a
// CTA (the pair's `side` 0 from the first row on, 1 from the last row on with A
// and C in each other's place and a negative row stride), N rows each.  Where
// they meet, x = y - P x' on either side (P the last C', x', P' and y' the
// other side's), so x = (I - P P')^{-1} (y - P y'); then both substitute back
// outwards.  Half the chain of block Thomas at the same arithmetic.  `sh`: the
// pair's exchange (kTwistShared).  Always guarded.
template <int M>
constexpr int kTwistShared = 2 * 32 * M + 32;  // doubles: 32 lanes x M values, then a flag a lane, of either side
template <class Num, int M, bool Reduced, bool Transposed = false, bool Twisted = false, bool Guard = Twisted>
__device__ __forceinline__ void thomas_cols_body(const double* A, const double* B, const double* C, double* D,
                                                 double* CW, size_t plane, ptrdiff_t rs, int N, bool raw,
                                                 unsigned long long* status, const ColLane& cl, double* Y = nullptr,
                                                 unsigned char* redo = nullptr, int side = 0, double* sh = nullptr,
                                                 int bar = 1) {
    static_assert(Guard || !Twisted, "elimination from both ends is guarded");
    using T = typename Num::T;
    using Acc = typename Num::Acc;
    const bool rhs = cl.j == M;
    const size_t col = (size_t)(rhs ? 0 : cl.j) * M * plane;
    const size_t in = Transposed ? (size_t)(rhs ? 0 : cl.j) * plane : col;  // this lane's column of an input block
    const size_t es = Transposed ? M * plane : plane, eb = Transposed && !rhs ? es : plane;
    const bool mat = cl.live && !rhs;
    const double* const pa = A + in;
    const double* const pb = rhs ? D : (Reduced ? A : B + in);
    const double* const pc = C + in;
    double* const yw = Guard ? Y : D;
    double* const pw = rhs ? yw : CW + col;
    unsigned bad = 0, amax = 0;
    [[maybe_unused]] float size = 0.f;  // of C'
    double va[M], vb[M], vc[M];
    T cp[M];
    // Raw inputs of row 0 (A_0 is not read).
    if constexpr (Reduced)
        col_load<M>(vb, pb, plane, cl.live && rhs);
    else
        col_load<M>(vb, pb, eb, cl.live);
    col_load<M>(vc, pc, es, mat && (Twisted || N > 1));
    for (int q = 0; q < N; ++q) {
        const ptrdiff_t o = q * rs;
        const bool last = q == N - 1;
        T a[M];
        Acc r[M], x[1][M];
#pragma unroll
        for (int i = 0; i < M; ++i) {
            if constexpr (Reduced)
                r[i] = rhs ? Num::acc(Num::from_raw(vb[i])) : Num::acc(i == cl.j ? Num::one() : Num::zero());
            else
                r[i] = Num::acc(Num::in_value(vb[i], rhs));
            if (q > 0) a[i] = Reduced ? Num::from_raw(va[i]) : Num::in_value(va[i], false);
            x[0][i] = Num::acc(Reduced ? Num::from_raw(vc[i]) : Num::in_value(vc[i], false));
        }
        // The next row's inputs, on their way while this row is eliminated.
        if (!last) {
            const ptrdiff_t p = o + rs;
            col_load<M>(va, pa + p, es, mat);
            if constexpr (Reduced)
                col_load<M>(vb, pb + p, plane, cl.live && rhs);
            else
                col_load<M>(vb, pb + p, eb, cl.live);
            col_load<M>(vc, pc + p, es, mat && (Twisted || q + 2 < N));
        }
        if (q > 0) col_product<Num, M>(r, a, cp, cl.base);
#pragma unroll
        for (int i = 0; i < M; ++i) x[0][i] = Num::asel(rhs, r[i], x[0][i]);
        col_gesv<Num, M, 1>(r, x, cl, bad);
#pragma unroll
        for (int i = 0; i < M; ++i) {
            cp[i] = Num::fin(x[0][i]);
            if constexpr (Guard) size = max_nan(size, Num::size(cp[i]));
        }
        if (cl.live && (Guard ? !last : rhs || !last)) {
#pragma unroll
            for (int i = 0; i < M; ++i) {
                double* const p = pw + o + (size_t)i * plane;
                if (rhs && last) amax = max(amax, Num::mag(cp[i]));
                if (Reduced || !Num::kConv || (rhs ? !last : raw))
                    Num::sts(p, cp[i]);
                else
                    Num::out(p, cp[i]);
            }
        }
    }
    bool keep = cl.live;
    if constexpr (Guard) {
        unsigned again = bad | (unsigned)(!rhs && Num::grown(size)), none = 0;
        col_merge<M>(again, none, cl);
        if constexpr (Twisted) {
            // This side's P and y (cp) and its outcome against the other's, lane by lane.
            const int lane = threadIdx.x & 31;
            double* const mine = sh + (side * 32 + lane) * M;
            const double* const other = sh + ((side ^ 1) * 32 + lane) * M;
            unsigned* const flags = reinterpret_cast<unsigned*>(sh + 2 * 32 * M) + lane;
#pragma unroll
            for (int i = 0; i < M; ++i) Num::sts(mine + i, cp[i]);
            flags[side * 32] = again;
            pair_barrier(bar);
            again |= flags[(side ^ 1) * 32];
            T oc[M];
            Acc r[M], x[1][M];
#pragma unroll
            for (int i = 0; i < M; ++i) {
                oc[i] = Num::lds(other + i);
                r[i] = rhs ? Num::acc(cp[i]) : Num::acc(i == cl.j ? Num::one() : Num::zero());
            }
            col_product<Num, M>(r, cp, oc, cl.base);
#pragma unroll
            for (int i = 0; i < M; ++i) x[0][i] = Num::asel(rhs, r[i], Num::acc0());
            col_gesv<Num, M, 1>(r, x, cl, bad);
#pragma unroll
            for (int i = 0; i < M; ++i) cp[i] = Num::fin(x[0][i]);
        }
        keep = cl.live && again == 0;
        if (keep && rhs) {
            double* const p = D + (N - 1) * rs;
#pragma unroll
            for (int i = 0; i < M; ++i) {
                amax = max(amax, Num::mag(cp[i]));
                Num::out(p + (size_t)i * plane, cp[i]);
            }
        }
    }
    // Backward: lane i < M computes x_q[i] = y_q[i] - sum over k of C'_q(i, k)
    // x_{q+1}[k]; the rows' values come kAhead rows ahead.
    constexpr int kAhead = cols_ahead<M>();
    T xn[M];
#pragma unroll
    for (int k = 0; k < M; ++k) xn[k] = col_bcast(cp[k], cl.base + M);
    const size_t mine = (size_t)(rhs ? 0 : cl.j) * plane;
    const double* const pr = CW + mine;  // row j of C'
    const double* const py = yw + mine;
    double* const px = D + mine;
    const bool back = keep && !rhs;
    double bc[kAhead][M], by[kAhead];
    auto fetch = [&](int slot, int q) {
        const bool on = back && q >= 0;
        const ptrdiff_t o = (q >= 0 ? q : 0) * rs;
        by[slot] = on ? py[o] : 0.0;
#pragma unroll
        for (int k = 0; k < M; ++k) bc[slot][k] = on ? pr[o + (size_t)(M * k) * plane] : 0.0;
    };
    // What the forward sweep stored is read back by other lanes of the group.
    __syncwarp();
#pragma unroll
    for (int s = 0; s < kAhead; ++s) fetch(s, N - 2 - s);
    for (int q0 = N - 2; q0 >= 0; q0 -= kAhead) {
#pragma unroll
        for (int s = 0; s < kAhead; ++s) {
            const int q = q0 - s;
            if (q >= 0) {
                const ptrdiff_t o = q * rs;
                Acc t = Num::acc(Num::from_raw(by[s]));
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    const T c = (Reduced || raw || !Num::kConv) ? Num::from_raw(bc[s][k])
                                                                : Num::in_value(bc[s][k], true);
                    Num::msub(t, c, xn[k]);
                }
                const T xq = Num::fin(t);
                fetch(s, q - kAhead);
                if (back) {
                    amax = max(amax, Num::mag(xq));
                    if (Reduced)
                        Num::sts(px + o, xq);
                    else
                        Num::out(px + o, xq);
                }
#pragma unroll
                for (int k = 0; k < M; ++k) xn[k] = col_bcast(xq, cl.base + k);
            }
        }
    }
    if constexpr (Twisted) {
        // The line's outcome, both sides together, reported by side 0.
        col_merge<M>(bad, amax, cl);
        unsigned* const u = reinterpret_cast<unsigned*>(sh) + 2 * (threadIdx.x & 31);
        pair_barrier(bar);  // the exchange has been read
        if (side == 1) {
            u[0] = bad;
            u[1] = amax;
        }
        pair_barrier(bar);
        if (side == 0 && cl.live && cl.j == 0) {
            if (keep)
                report_status(status, bad | u[0] | range_bits<Num>(max(amax, u[1]), true));
            else
                *redo = 1;
        }
    } else {
        if (Guard && cl.live && !keep && cl.j == 0) *redo = 1;
        ColLane out = cl;
        out.live = keep;
        col_report<Num, M>(status, bad, amax, true, out);
    }
}

// CTAs of four warps an SM holds (the register cap).
template <int M>
__host__ __device__ constexpr int cols_min_ctas(bool local_stage) {
    return M <= (local_stage ? 4 : 6) ? 4 : (local_stage && M > 6 ? 2 : 3);
}
// Warps an SM holds of the single-segment kernels.
template <int M>
__host__ __device__ constexpr int cols_warps() {
    return 4 * cols_min_ctas<M>(false);
}
template <class Num, int M, bool Guard>
__global__ void __launch_bounds__(32 * cols_warps<M>(), 1) k_thomas_cols(const SolveArgs g, const LineStrides ls,
                                                                       unsigned char* redo) {
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const long long s = cl.live ? cl.sys : 0;
    const size_t o = (size_t)(s % ls.lin) * (size_t)ls.in + (size_t)(s / ls.lin) * (size_t)ls.out;
    thomas_cols_body<Num, M, false, false, false, Guard>(g.a + o, g.b + o, g.c + o, g.d + o, g.cw + o, (size_t)ls.elem,
                                                         (size_t)ls.row, g.nrow, g.factors_raw != 0, g.status, cl,
                                                         Guard ? g.aw + o : nullptr, Guard ? redo + s : nullptr);
}

template <class Num, int M>
__global__ void __launch_bounds__(128, cols_min_ctas<M>(false)) k_reduced_cols(const SolveArgs g) {
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const size_t s = cl.live ? (size_t)cl.sys : 0, rs = (size_t)g.nsys;
    thomas_cols_body<Num, M, true>(g.ra + s, nullptr, g.rc + s, g.rd + s, g.rc + s, rs * 2 * g.nseg, rs, 2 * g.nseg,
                                   true, g.status, cl);
}

// M^T lambda = g for the adjoint, from the forward blocks as they are stored:
// At_q = C_{q-1}^T, Bt_q = B_q^T, Ct_q = A_{q+1}^T; lambda in D, the factors in
// the workspace (raw).
template <class Num, int M, bool Guard>
__global__ void __launch_bounds__(32 * cols_warps<M>(), 1) k_transposed_cols(const SolveArgs g, unsigned char* redo) {
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const size_t s = cl.live ? (size_t)cl.sys : 0, rs = (size_t)g.nsys;
    thomas_cols_body<Num, M, false, true, false, Guard>(g.c + s - rs, g.b + s, g.a + s + rs, g.d + s, g.cw + s,
                                                        rs * g.nrow, rs, g.nrow, true, g.status, cl,
                                                        Guard ? g.aw + s : nullptr, Guard ? redo + s : nullptr);
}

// The twisted solve, one pair of warps a CTA; Transposed: of M^T, as above.
template <class Num, int M, bool Transposed>
__global__ void __launch_bounds__(64, 2 * cols_min_ctas<M>(false)) k_twist_cols(const SolveArgs g, unsigned char* redo) {
    __shared__ double sh[kTwistShared<M>];
    const ColLane cl = col_lane<M>(g.nsys, blockIdx.x);
    const int side = threadIdx.x >> 5, n0 = g.nrow / 2, n = side ? g.nrow - n0 : n0;
    const ptrdiff_t rs = g.nsys, s = cl.live ? (ptrdiff_t)cl.sys : 0;
    const size_t plane = (size_t)g.nsys * g.nrow;
    const ptrdiff_t o = s + (side ? rs * (g.nrow - 1) : 0);
    const double* const a = Transposed ? g.c - rs : g.a;  // row q of the lower blocks at a + o + q * rs
    const double* const c = Transposed ? g.a + rs : g.c;
    thomas_cols_body<Num, M, false, Transposed, true>((side ? c : a) + o, g.b + o, (side ? a : c) + o, g.d + o,
                                                      g.cw + o, plane, side ? -rs : rs, n, true, g.status, cl, g.aw + o,
                                                      redo + s, side, sh);
}

// Local stage of one segment of one system per group (modi_body, column per
// lane): lane j < M carries column j of A' and C', lane M d' (in the place of
// a C' column).  Pointers at system 0, rows rs apart, 2 * nseg reduced rows rs
// apart too; segment rows f .. f + n - 1.  Transposed: A_q, B_q, C_q are
// C_{q-1}^T, B_q^T, A_{q+1}^T of the blocks in C, B, A (zero past the ends).
template <class Num, int M, bool Transposed>
__device__ __forceinline__ void modi_cols_body(const double* A, const double* B, const double* C, double* D, double* AW,
                                               double* CW, double* RA, double* RC, double* RD, size_t rs, int nrow,
                                               int nseg, int seg, bool raw, unsigned long long* status,
                                               const ColLane& cl) {
    using T = typename Num::T;
    using Acc = typename Num::Acc;
    const bool rhs = cl.j == M, mat = cl.live && !rhs;
    int f, l;
    seg_rows(nrow, nseg, seg, f, l);
    const int n = l - f + 1;
    const size_t plane = rs * nrow, s = cl.live ? (size_t)cl.sys : 0;
    const size_t fo = (size_t)f * rs + s, col = (size_t)(rhs ? 0 : cl.j) * M * plane;
    const size_t in = Transposed ? (size_t)(rhs ? 0 : cl.j) * plane : col;  // this lane's column of an input block
    const size_t es = Transposed ? M * plane : plane, eb = Transposed && !rhs ? es : plane;
    const double* const pa = (Transposed ? C - rs : A) + fo + in;
    const double* const pb = rhs ? D + fo : B + fo + in;
    const double* const pc = (Transposed ? A + rs : C) + fo + in;
    double* const qa = AW + fo + col;
    double* const qc = rhs ? D + fo : CW + fo + col;
    const size_t rplane = rs * 2 * nseg, rcol = (size_t)(rhs ? 0 : cl.j) * M * rplane;
    double* const ra = RA + s + rcol;
    double* const rc = rhs ? RD + s : RC + s + rcol;
    const bool no_a = Transposed && f == 0;  // the line's first row has no A^T, its last no C^T
    auto load = [&](double (&va)[M], double (&vb)[M], double (&vc)[M], int q) {
        const size_t o = (size_t)q * rs;
        col_load<M>(va, pa + o, es, mat && !(no_a && q == 0));
        col_load<M>(vb, pb + o, eb, cl.live);
        col_load<M>(vc, pc + o, es, mat && !(Transposed && f + q == nrow - 1));
    };
    unsigned bad = 0;
    // This lane's column of row q into the factor arrays, and into the
    // reduced row rr (rr < 0: none).
    auto store = [&](int q, const T (&ap)[M], const T (&cp)[M], int rr) {
        if (!cl.live) return;
        const size_t o = (size_t)q * rs;
#pragma unroll
        for (int i = 0; i < M; ++i) {
            if (!rhs) st_fac<Num>(qa + o + (size_t)i * plane, ap[i], raw);
            st_fac<Num>(qc + o + (size_t)i * plane, cp[i], raw || rhs);
            if (rr >= 0) {
                const size_t ro = (size_t)rr * rs + (size_t)i * rplane;
                if (!rhs) Num::sts(ra + ro, ap[i]);
                Num::sts(rc + ro, cp[i]);
            }
        }
    };
    auto fac = [&](double v) -> T {  // a factor read back (d' is always raw)
        return (raw || !Num::kConv || rhs) ? Num::from_raw(v) : Num::in_value(v, true);
    };
    T ap[M], cp[M];
    {
        double va[M], vb[M], vc[M];
        load(va, vb, vc, 0);
        for (int q = 0; q < n; ++q) {
            T a[M];
            Acc r[M], x[2][M];
#pragma unroll
            for (int i = 0; i < M; ++i) {
                a[i] = Num::in_value(va[i], false);
                r[i] = Num::acc(Num::in_value(vb[i], rhs));
                x[0][i] = (q < 2) ? Num::acc(a[i]) : Num::acc0();
                x[1][i] = Num::acc(Num::in_value(vc[i], false));
            }
            if (q + 1 < n) load(va, vb, vc, q + 1);
            if (q >= 2) col_product2<Num, M>(r, x[0], a, cp, ap, cl.base);
#pragma unroll
            for (int i = 0; i < M; ++i) x[1][i] = Num::asel(rhs, r[i], x[1][i]);
            col_gesv<Num, M, 2>(r, x, cl, bad);
#pragma unroll
            for (int i = 0; i < M; ++i) {
                ap[i] = Num::fin(x[0][i]);
                cp[i] = Num::fin(x[1][i]);
            }
            store(q, ap, cp, q == n - 1 ? 2 * seg + 1 : -1);
        }
    }
    // Backward, rows n-3 .. 1, carried row q + 1; then row 0 with R = I -
    // C'_0 A'_1.  Every lane reads back only what it stored.
    {
        const int q1 = (n >= 4) ? n - 2 : 1;
        double va[M], vc[M];
        col_load<M>(va, qa + (size_t)q1 * rs, plane, mat);
        col_load<M>(vc, qc + (size_t)q1 * rs, plane, cl.live);
#pragma unroll
        for (int i = 0; i < M; ++i) {
            ap[i] = fac(va[i]);
            cp[i] = fac(vc[i]);
        }
        const int first = (n >= 4) ? n - 3 : 0;
        col_load<M>(va, qa + (size_t)first * rs, plane, mat);
        col_load<M>(vc, qc + (size_t)first * rs, plane, cl.live);
        for (int q = first; q >= 0; --q) {
            T c[M];
            Acc x[2][M];
#pragma unroll
            for (int i = 0; i < M; ++i) {
                c[i] = fac(vc[i]);
                x[0][i] = Num::acc(fac(va[i]));
                x[1][i] = rhs ? Num::acc(c[i]) : Num::acc0();
            }
            if (q > 0) {
                col_load<M>(va, qa + (size_t)(q - 1) * rs, plane, mat);
                col_load<M>(vc, qc + (size_t)(q - 1) * rs, plane, cl.live);
                col_product2<Num, M>(x[0], x[1], c, ap, cp, cl.base);
            } else {
                Acc r[M];
#pragma unroll
                for (int i = 0; i < M; ++i) r[i] = Num::acc(i == cl.j ? Num::one() : Num::zero());
                col_product2<Num, M>(r, x[1], c, ap, cp, cl.base);
                col_gesv<Num, M, 2>(r, x, cl, bad);
            }
#pragma unroll
            for (int i = 0; i < M; ++i) {
                ap[i] = Num::fin(x[0][i]);
                cp[i] = Num::fin(x[1][i]);
            }
            store(q, ap, cp, q == 0 ? 2 * seg : -1);
        }
    }
    col_report<Num, M>(status, bad, 0u, false, cl);
}
template <class Num, int M>
__global__ void __launch_bounds__(128, cols_min_ctas<M>(true)) k_modi_cols(const SolveArgs g) {
    modi_cols_body<Num, M, false>(g.a, g.b, g.c, g.d, g.aw, g.cw, g.ra, g.rc, g.rd, (size_t)g.nsys, g.nrow, g.nseg,
                                  blockIdx.y, g.factors_raw != 0, g.status, col_lane<M>(g.nsys, grid_warp()));
}

// The two-stage method for the flagged lines of one group (the arithmetic and
// the outcome that a plan in segments has): a CTA's warps take segments, the
// first one the reduced systems, all threads pieces of the update.  Pointers at
// system 0 of `nsys`, rows rs apart; with `saved` d is in AW's first planes, else
// still in D; flags are cleared.  Returns at once where no line of the group is
// flagged.
template <class Num, int M, bool Transposed>
__device__ __forceinline__ void redo_cols_group(const double* A, const double* B, const double* C, double* D, double* AW,
                                                double* CW, double* RA, double* RC, double* RD, size_t rs, int nsys,
                                                int nrow, int nseg, long long group, unsigned char* redo, bool saved,
                                                unsigned long long* status) {
    constexpr int S = cols_systems<M>();
    ColLane cl = col_lane<M>(nsys, group);
    cl.live = cl.live && redo[cl.sys] != 0;
    if (!__syncthreads_or(cl.live)) return;
    const int per = blockDim.x / S, part = threadIdx.x / S;  // rows or pieces at a time
    const long long sys = group * S + threadIdx.x % S;
    const bool mine = part < per && sys < nsys && redo[sys] != 0;
    if (saved && mine) {
        for (long long r = part; r < (long long)M * nrow; r += per)
            D[(size_t)r * rs + (size_t)sys] = AW[(size_t)r * rs + (size_t)sys];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int seg = warp; seg < nseg; seg += warps)
        modi_cols_body<Num, M, Transposed>(A, B, C, D, AW, CW, RA, RC, RD, rs, nrow, nseg, seg, true, status, cl);
    __syncthreads();
    if (warp == 0) {
        const size_t s = cl.live ? (size_t)cl.sys : 0;
        thomas_cols_body<Num, M, true>(RA + s, nullptr, RC + s, RD + s, RC + s, rs * 2 * nseg, (ptrdiff_t)rs, 2 * nseg,
                                       true, status, cl);
    }
    __syncthreads();
    unsigned amax = 0;
    if (mine) {
        const int pieces = ((nrow + nseg - 1) / nseg + kUpdateRows - 1) / kUpdateRows;
        for (long long u = part; u < (long long)nseg * pieces; u += per) {
            const int seg = (int)(u / pieces), q0 = (int)(u % pieces) * kUpdateRows;
            int f, l;
            seg_rows(nrow, nseg, seg, f, l);
            const int n = l - f + 1, q1 = min(n, q0 + kUpdateRows);
            const size_t o = (size_t)f * rs + (size_t)sys;
            if (q0 < n)
                update_rows<Num, M, true>(AW + o, CW + o, D + o, rs * nrow, rs, n, q0, q1, RD + sys, rs * 2 * nseg, rs,
                                          seg, amax);
        }
    }
    report_status(status, range_bits<Num>(amax, false));
    __syncthreads();
    if (mine && part == 0) redo[sys] = 0;
}
// One CTA a group: where nothing is flagged, 3.5 us a launch of 1544 CTAs.
template <class Num, int M, bool Transposed>
__global__ void __launch_bounds__(128, cols_min_ctas<M>(true)) k_redo_cols(const SolveArgs g, unsigned char* redo,
                                                                             bool saved) {
    redo_cols_group<Num, M, Transposed>(g.a, g.b, g.c, g.d, g.aw, g.cw, g.ra, g.rc, g.rd, (size_t)g.nsys, g.nsys,
                                        g.nrow, g.nseg, blockIdx.x, redo, saved, g.status);
}

// CTA of the local stage and the reduced solve: one warp while there are fewer
// than eight warps an SM (they spread over the SMs), else four, whose
// neighbouring systems share their 32-byte sectors in L1.
template <int M>
inline int cols_threads(const SolveArgs& g, int segs) {
    if (!g.tpb_auto) return g.tpb;
    const long long warps = ((long long)g.nsys + cols_systems<M>() - 1) / cols_systems<M>() * segs;
    return warps < 8LL * (g.sms > 0 ? g.sms : 1) ? 32 : 128;
}
// CTA of the single-segment kernels: an SM's even share of the warps, or of a
// round of them where they are not resident together, so that no SM runs longer
// than another.  In CTAs of four, nine warps an SM made twelve on some, and past
// residency the first SMs to finish took the rest of the batch between them.
// FP64, 128 rows: m = 8, 9 warps an SM (4104 systems) 3840 -> 3080 us, 12.5
// (5700) 7480 -> 4550, 17 7540 -> 6140; m = 5, 9 1675 -> 1358, 12.5 2212 ->
// 1887.  Float-float up to m = 5 in one round: 7 warps 443 -> 424, 12.5 771 ->
// 695; its blocks past m = 5 (m = 8, 10 warps 1294 -> 1321) and further rounds
// (m = 5, 17 warps 984 -> 1017) are better off in fours, whose code and sectors
// stay in L1 while the fours take turns.
template <class Num, int M>
inline int cols_threads_even(const SolveArgs& g) {
    if (!g.tpb_auto) return g.tpb;
    const long long n = g.sms > 0 ? g.sms : 1, warps = ((long long)g.nsys + cols_systems<M>() - 1) / cols_systems<M>();
    const long long even = (warps + n - 1) / n, rounds = (even + cols_warps<M>() - 1) / cols_warps<M>();
    if (Num::kConv && (M > 5 || rounds > 1)) return cols_threads<M>(g, 1);
    return 32 * (int)((even + rounds - 1) / rounds);
}
template <int M>
inline unsigned cols_grid(int nsys, int tpb) {
    const long long per = (long long)cols_systems<M>() * (tpb / 32);
    return (unsigned)((nsys + per - 1) / per);
}

template <class Num, int M>
cudaError_t launch_thomas_cols(const SolveArgs& g, const LineStrides& ls, unsigned char* redo) {
    const int tpb = cols_threads_even<Num, M>(g);
    const auto kernel = redo ? k_thomas_cols<Num, M, true> : k_thomas_cols<Num, M, false>;
    kernel<<<cols_grid<M>(g.nsys, tpb), tpb, 0, g.stream>>>(g, ls, redo);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_twist_cols(const SolveArgs& g, unsigned char* redo) {
    k_twist_cols<Num, M, false><<<cols_grid<M>(g.nsys, 32), 64, 0, g.stream>>>(g, redo);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_transposed_cols(const SolveArgs& g, int twisted, unsigned char* redo) {
    const int tpb = twisted ? 64 : cols_threads_even<Num, M>(g);
    const auto kernel = twisted ? k_twist_cols<Num, M, true>
                                : (redo ? k_transposed_cols<Num, M, true> : k_transposed_cols<Num, M, false>);
    kernel<<<cols_grid<M>(g.nsys, twisted ? 32 : tpb), tpb, 0, g.stream>>>(g, redo);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_redo_cols(const SolveArgs& g, int transposed, unsigned char* redo, bool saved) {
    const auto kernel = transposed ? k_redo_cols<Num, M, true> : k_redo_cols<Num, M, false>;
    kernel<<<cols_grid<M>(g.nsys, 32), 128, 0, g.stream>>>(g, redo, saved);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_modi_cols(const SolveArgs& g) {
    const int tpb = cols_threads<M>(g, g.nseg);
    k_modi_cols<Num, M><<<dim3(cols_grid<M>(g.nsys, tpb), (unsigned)g.nseg), tpb, 0, g.stream>>>(g);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_reduced_cols(const SolveArgs& g) {
    const int tpb = cols_threads<M>(g, 1);
    k_reduced_cols<Num, M><<<cols_grid<M>(g.nsys, tpb), tpb, 0, g.stream>>>(g);
    return cudaGetLastError();
}

}  // namespace pbt

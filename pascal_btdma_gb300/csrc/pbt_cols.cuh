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
// Twisted: the line is eliminated from both ends at once, by two warps of a
// CTA (the pair's `side` 0 from the first row on, 1 from the last row on with A
// and C in each other's place and a negative row stride), N rows each.  Where
// they meet, x = y - P x' on either side (P the last C', x', P' and y' the
// other side's), so x = (I - P P')^{-1} (y - P y'); then both substitute back
// outwards.  Half the chain of block Thomas at the same arithmetic.  `sh`: the
// pair's exchange, 2 x 32 lanes x M values.
template <class Num, int M, bool Reduced, bool Transposed = false, bool Twisted = false>
__device__ __forceinline__ void thomas_cols_body(const double* A, const double* B, const double* C, double* D,
                                                 double* CW, size_t plane, ptrdiff_t rs, int N, bool raw,
                                                 unsigned long long* status, const ColLane& cl, int side = 0,
                                                 double* sh = nullptr, int bar = 1) {
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
    double* const pw = rhs ? D : CW + col;
    unsigned bad = 0, amax = 0;
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
        for (int i = 0; i < M; ++i) cp[i] = Num::fin(x[0][i]);
        if (cl.live && (Twisted ? !last : rhs || !last)) {
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
    if constexpr (Twisted) {
        // This side's P and y (cp) against the other's, lane by lane.
        double* const mine = sh + (side * 32 + (threadIdx.x & 31)) * M;
        const double* const other = sh + ((side ^ 1) * 32 + (threadIdx.x & 31)) * M;
#pragma unroll
        for (int i = 0; i < M; ++i) Num::sts(mine + i, cp[i]);
        pair_barrier(bar);
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
        const ptrdiff_t o = (N - 1) * rs;
#pragma unroll
        for (int i = 0; i < M; ++i) {
            cp[i] = Num::fin(x[0][i]);
            if (cl.live && rhs) {
                amax = max(amax, Num::mag(cp[i]));
                Num::out(pw + o + (size_t)i * plane, cp[i]);
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
    double* const py = D + mine;
    double bc[kAhead][M], by[kAhead];
    auto fetch = [&](int slot, int q) {
        const bool on = mat && q >= 0;
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
                if (mat) {
                    amax = max(amax, Num::mag(xq));
                    if (Reduced)
                        Num::sts(py + o, xq);
                    else
                        Num::out(py + o, xq);
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
        if (side == 0 && cl.live && cl.j == 0)
            report_status(status, bad | u[0] | range_bits<Num>(max(amax, u[1]), true));
    } else {
        col_report<Num, M>(status, bad, amax, true, cl);
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
template <class Num, int M>
__global__ void __launch_bounds__(32 * cols_warps<M>(), 1) k_thomas_cols(const SolveArgs g, const LineStrides ls) {
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const long long s = cl.live ? cl.sys : 0;
    const size_t o = (size_t)(s % ls.lin) * (size_t)ls.in + (size_t)(s / ls.lin) * (size_t)ls.out;
    thomas_cols_body<Num, M, false>(g.a + o, g.b + o, g.c + o, g.d + o, g.cw + o, (size_t)ls.elem, (size_t)ls.row,
                                    g.nrow, g.factors_raw != 0, g.status, cl);
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
template <class Num, int M>
__global__ void __launch_bounds__(32 * cols_warps<M>(), 1) k_transposed_cols(const SolveArgs g) {
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const size_t s = cl.live ? (size_t)cl.sys : 0, rs = (size_t)g.nsys;
    thomas_cols_body<Num, M, false, true>(g.c + s - rs, g.b + s, g.a + s + rs, g.d + s, g.cw + s, rs * g.nrow, rs,
                                          g.nrow, true, g.status, cl);
}

// The twisted solve, one pair of warps a CTA; Transposed: of M^T, as above.
template <class Num, int M, bool Transposed>
__global__ void __launch_bounds__(64, 2 * cols_min_ctas<M>(false)) k_twist_cols(const SolveArgs g) {
    __shared__ double sh[2 * 32 * M];
    const ColLane cl = col_lane<M>(g.nsys, blockIdx.x);
    const int side = threadIdx.x >> 5, n0 = g.nrow / 2, n = side ? g.nrow - n0 : n0;
    const ptrdiff_t rs = g.nsys;
    const size_t plane = (size_t)g.nsys * g.nrow;
    const ptrdiff_t o = (cl.live ? (ptrdiff_t)cl.sys : 0) + (side ? rs * (g.nrow - 1) : 0);
    const double* const a = Transposed ? g.c - rs : g.a;  // row q of the lower blocks at a + o + q * rs
    const double* const c = Transposed ? g.a + rs : g.c;
    thomas_cols_body<Num, M, false, Transposed, true>((side ? c : a) + o, g.b + o, (side ? a : c) + o, g.d + o,
                                                      g.cw + o, plane, side ? -rs : rs, n, true, g.status, cl, side, sh);
}

// Local stage of one segment of one system per group (modi_body, column per
// lane): lane j < M carries column j of A' and C', lane M d' (in the place of
// a C' column).
template <class Num, int M>
__global__ void __launch_bounds__(128, cols_min_ctas<M>(true)) k_modi_cols(const SolveArgs g) {
    using T = typename Num::T;
    using Acc = typename Num::Acc;
    const ColLane cl = col_lane<M>(g.nsys, grid_warp());
    const bool rhs = cl.j == M, mat = cl.live && !rhs, raw = g.factors_raw != 0;
    const int seg = blockIdx.y;
    int f, l;
    seg_rows(g.nrow, g.nseg, seg, f, l);
    const int n = l - f + 1;
    const size_t rs = (size_t)g.nsys, plane = rs * g.nrow, s = cl.live ? (size_t)cl.sys : 0;
    const size_t fo = (size_t)f * rs + s, col = (size_t)(rhs ? 0 : cl.j) * M * plane;
    const double* const pa = g.a + fo + col;
    const double* const pb = rhs ? g.d + fo : g.b + fo + col;
    const double* const pc = g.c + fo + col;
    double* const qa = g.aw + fo + col;
    double* const qc = rhs ? g.d + fo : g.cw + fo + col;
    const size_t rplane = rs * 2 * g.nseg, rcol = (size_t)(rhs ? 0 : cl.j) * M * rplane;
    double* const ra = g.ra + s + rcol;
    double* const rc = rhs ? g.rd + s : g.rc + s + rcol;
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
        col_load<M>(va, pa, plane, mat);
        col_load<M>(vb, pb, plane, cl.live);
        col_load<M>(vc, pc, plane, mat);
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
            if (q + 1 < n) {
                const size_t p = (size_t)(q + 1) * rs;
                col_load<M>(va, pa + p, plane, mat);
                col_load<M>(vb, pb + p, plane, cl.live);
                col_load<M>(vc, pc + p, plane, mat);
            }
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
    col_report<Num, M>(g.status, bad, 0u, false, cl);
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
cudaError_t launch_thomas_cols(const SolveArgs& g, const LineStrides& ls) {
    const int tpb = cols_threads_even<Num, M>(g);
    k_thomas_cols<Num, M><<<cols_grid<M>(g.nsys, tpb), tpb, 0, g.stream>>>(g, ls);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_twist_cols(const SolveArgs& g) {
    k_twist_cols<Num, M, false><<<cols_grid<M>(g.nsys, 32), 64, 0, g.stream>>>(g);
    return cudaGetLastError();
}
template <class Num, int M>
cudaError_t launch_transposed_cols(const SolveArgs& g, int twisted) {
    if (twisted) {
        k_twist_cols<Num, M, true><<<cols_grid<M>(g.nsys, 32), 64, 0, g.stream>>>(g);
        return cudaGetLastError();
    }
    const int tpb = cols_threads_even<Num, M>(g);
    k_transposed_cols<Num, M><<<cols_grid<M>(g.nsys, tpb), tpb, 0, g.stream>>>(g);
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

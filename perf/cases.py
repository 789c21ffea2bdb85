"""The work that users of this solver have it do, as cases that can be timed.

A case is a dict of plain values; `prepare` makes what a program has in hand
before the call (device arrays, the plan), `run` is one pass through the
public entry points, `exact` the same result in 64 bits by plain torch.

Kinds of case:
  solve    solve_noncyclic / solve_cyclic on a uniform batch (any precision)
  grad     BlockTridiagonalSolve forward and backward (autograd)
  batch    BatchPlan: systems of uneven length and mixed block size
  heat     SharedMatrix: constant-coefficient ADI step in a haloed 3-D field
  lines    solve_noncyclic_lines: sweeps in an application's own 3-D arrays

Systems are A_q x_{q-1} + B_q x_q + C_q x_{q+1} = d_q with A, C, R and d iid
uniform in [-1, 1) and B = R + diag(delta * rowsum(|A| + |C| + |R|)), the
diagonally dominant blocks of implicit schemes.  A time step refills the
right-hand side, which the solves overwrite; `run` does that with a copy.
"""
import torch

import pascal_btdma_gb300 as pbt
from pascal_btdma_gb300 import batch as pbatch
from pascal_btdma_gb300 import shared as pshared

DEV = "cuda"
F64 = torch.float64
# Elements of A in the largest uniform cases: 65536 lines of 256 rows at m = 5,
# and 4096 lines of 1024 rows at m = 8, for the block sizes above 6.
MOST = 65536 * 256 * 25
MOST_WIDE = 4096 * 1024 * 64


def _solve(name, m, nsys, nrow, nseg, precision, delta=1.2, cyclic=False, scaled=False):
    return {"name": name, "kind": "solve", "m": m, "nsys": nsys, "nrow": nrow, "nseg": nseg, "precision": precision,
            "delta": delta, "cyclic": cyclic, "scaled": scaled}


def listed():
    return [
        # The reference's sample run on four ranks, in its own arithmetic: a
        # small batch, all latency and launches.
        _solve("sample_m3_p4_fp64", 3, 1024, 128, 4, "fp64", delta=2.0),
        # Odd sizes everywhere, lines split in three: ordinary work of a
        # middle-sized 2-D problem in the fast arithmetic.
        _solve("ragged_m3_p3_ff", 3, 12347, 301, 3, "ff"),
        # The production pencil batch of a 3-D Euler solver (256 x 256 lines),
        # in the fast arithmetic, in the default one, and refined to 1e-12 with
        # badly scaled rows.
        _solve("pencil_m5_ff", 5, 65536, 256, 1, "ff"),
        _solve("pencil_m5_fp64", 5, 65536, 256, 1, "fp64"),
        _solve("pencil_m5_refine", 5, 65536, 256, 1, "fp32_refine", delta=1.5, scaled=True),
        # The same lines in a periodic box.
        _solve("periodic_m5_ff", 5, 65536, 256, 1, "ff", cyclic=True),
        # Few, very long lines: the two-stage method with many segments.
        _solve("long_m4_p128_ff", 4, 256, 32768, 128, "ff"),
        # The largest block size of the reference's study (64 x 64 x 1024, m = 8)
        # in the default arithmetic.
        _solve("study_m8_fp64", 8, 4096, 1024, 4, "fp64"),
        # A differentiable solver layer: forward and all gradients, lines in
        # eight segments.
        {"name": "grad_m4_p8_fp64", "kind": "grad", "m": 4, "nsys": 16384, "nrow": 512, "nseg": 8, "precision": "fp64",
         "delta": 1.5},
        # Thousands of systems of different length and block size in one call.
        {"name": "uneven_m2to5_ff", "kind": "batch", "nsys": 32768, "nmin": 16, "nmax": 4096, "mmin": 2, "mmax": 5,
         "shapes": 1, "seg_len": 64, "precision": "ff", "delta": 1.5},
        # One ADI step of a heat equation: three sweeps with one matrix in a
        # 512^3 field with a halo of 2, in place.
        {"name": "heat3d_512_ff", "kind": "heat", "n": 512, "halo": 2, "sigma": 0.05, "precision": "ff"},
        # One ADI step of a 3-D Euler solver in its own arrays: a sweep along
        # each axis of a 256^3 field, the contiguous one among them.
        {"name": "euler3d_xyz_m5_ff", "kind": "lines", "m": 5, "n1": 256, "n2": 256, "n3": 256, "sweeps": "xyz",
         "precision": "ff", "delta": 1.2},
    ]


def _spread(rng, lo, hi):
    """An integer, log-uniform in [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "grad", "batch", "heat", "lines"])
    if kind == "solve":
        m = rng.randint(2, 8)
        nrow = _spread(rng, 16, 32768)
        nsys = _spread(rng, 64, max(64, min(65536, (MOST if m <= 6 else MOST_WIDE) // (nrow * m * m))))
        # Segments of 16 to 512 rows, as a program run on several ranks has them.
        nseg = max(1, nrow // _spread(rng, 16, 512))
        cyclic = rng.random() < 0.25
        precision = rng.choice(["fp64", "ff"] if cyclic else ["fp64", "ff", "ff", "fp32_refine"])
        if precision == "fp32_refine":
            m = min(m, 6)
        return {"kind": "solve", "m": m, "nsys": nsys, "nrow": nrow, "nseg": nseg, "precision": precision,
                "delta": rng.choice([1.05, 1.2, 1.5, 2.0]), "cyclic": cyclic, "scaled": precision == "fp32_refine"}
    if kind == "grad":
        m = rng.randint(2, 6)
        nrow = _spread(rng, 16, 1024)
        nsys = _spread(rng, 64, min(65536, 16384 * 512 * 16 // (nrow * m * m)))
        return {"kind": "grad", "m": m, "nsys": nsys, "nrow": nrow, "nseg": max(1, nrow // _spread(rng, 16, 512)),
                "precision": rng.choice(["fp64", "ff"]), "delta": 1.5}
    if kind == "batch":
        mmin = rng.randint(1, 4)
        nmin = _spread(rng, 4, 128)
        return {"kind": "batch", "nsys": _spread(rng, 256, 32768), "nmin": nmin, "nmax": _spread(rng, 2 * nmin, 4096),
                "mmin": mmin, "mmax": rng.randint(mmin, 5), "shapes": rng.randint(1, 1 << 20),
                "seg_len": rng.choice([32, 64, 128, 256]),
                "precision": rng.choice(["fp64", "ff"]), "delta": 1.5}
    if kind == "heat":
        return {"kind": "heat", "n": 2 * _spread(rng, 16, 256), "halo": 2, "sigma": rng.choice([0.02, 0.05, 0.2]),
                "precision": rng.choice(["fp64", "ff"])}
    n = [_spread(rng, 16, 256) for _ in range(3)]
    return {"kind": "lines", "m": rng.randint(2, 6) if max(n) < 200 else rng.randint(2, 5), "n1": n[0], "n2": n[1],
            "n3": n[2], "sweeps": rng.choice(["x", "y", "z", "xyz"]), "precision": rng.choice(["fp64", "ff"]),
            "delta": rng.choice([1.05, 1.2, 1.5])}


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _uniform(shape, g):
    return torch.rand(shape, dtype=F64, device=DEV, generator=g).mul_(2.0).sub_(1.0)


def _blocks(m, rows, delta, g, scaled=False):
    """A, B, C [j, i, *rows] and d [i, *rows]: element (i, j) of a block at
    [j, i], the reference layout with rows = (nrow, nsys)."""
    A, C, B = (_uniform((m, m) + rows, g) for _ in range(3))
    d = _uniform((m,) + rows, g)
    for i in range(m):
        s = torch.zeros(rows, dtype=F64, device=DEV)
        for j in range(m):
            s += A[j, i].abs()
            s += C[j, i].abs()
            s += B[j, i].abs()
        B[i, i] += delta * s
    if scaled:  # each block row times a log-uniform factor in [1e-3, 1e3]
        f = torch.pow(10.0, 3.0 * _uniform(rows, g))
        for x in (A, B, C, d):
            x *= f
    return A, B, C, d


def _solve_inputs(case, seed):
    A, B, C, d = _blocks(case["m"], (case["nrow"], case["nsys"]), case["delta"], _gen(seed), case.get("scaled", False))
    if not case.get("cyclic", False):
        A[:, :, 0] = 0.0
        C[:, :, -1] = 0.0
    return A, B, C, d


def _uneven_shapes(case):
    """(m, n) per system, which the case alone fixes: n log-uniform in [nmin,
    nmax], m uniform."""
    g = torch.Generator()
    g.manual_seed(104729 * case["shapes"] + 7)
    u = torch.rand(case["nsys"], dtype=F64, generator=g)
    n = (case["nmin"] * (case["nmax"] / case["nmin"]) ** u).round().long().clamp(case["nmin"], case["nmax"])
    m = torch.randint(case["mmin"], case["mmax"] + 1, (case["nsys"],), generator=g)
    return m, n


def _batch_inputs(case, seed):
    """Per-system arrays: system s is the reference layout of one system at its
    own offset.  Returns m, n, the user arrays, and per block size the index
    maps (systems, their n, matrix and vector indices of every element)."""
    m, n = _uneven_shapes(case)
    mo = torch.cumsum(n * m * m, 0) - n * m * m
    vo = torch.cumsum(n * m, 0) - n * m
    g = _gen(seed)
    tot_m, tot_v = int((n * m * m).sum()), int((n * m).sum())
    user = [torch.empty(tot_m, dtype=F64, device=DEV) for _ in range(3)] + [torch.empty(tot_v, dtype=F64, device=DEV)]
    groups = {}
    for mm in range(case["mmin"], case["mmax"] + 1):
        sel = (m == mm).nonzero().flatten()
        if not sel.numel():
            continue
        ns = n[sel].to(DEV)
        start = torch.cumsum(ns, 0) - ns
        rows = int(ns.sum())
        sysi = torch.repeat_interleave(torch.arange(sel.numel(), device=DEV), ns)
        q = torch.arange(rows, device=DEV) - start[sysi]
        nn = ns[sysi]
        mat0, vec0 = mo[sel].to(DEV)[sysi] + q, vo[sel].to(DEV)[sysi] + q
        A, B, C, d = _blocks(mm, (rows,), case["delta"], g)
        A[:, :, q == 0] = 0.0
        C[:, :, q == nn - 1] = 0.0
        for j in range(mm):
            for i in range(mm):
                at = mat0 + nn * (i + mm * j)
                for u, x in zip(user, (A, B, C)):
                    u[at] = x[j, i]
        for i in range(mm):
            user[3][vec0 + nn * i] = d[i]
        groups[mm] = (sel.to(DEV), ns, start, A, B, C, d, vec0, nn)
    return m, n, user, groups


def _heat_field(case, seed):
    k = case["n"] + 2 * case["halo"]
    return torch.rand((k, k, k), dtype=F64, device=DEV, generator=_gen(seed))


def _heat_lines(case, interior, axis):
    st, n = interior.stride(), case["n"]
    outer, inner = [a for a in range(3) if a != axis]
    return pshared.Lines(n, n, st[inner], st[outer], 2 * st[axis], st[axis])


def _field_inputs(case, seed):
    """A, B, C [j, i, k3, k2, k1] and d of a 3-D field, index 1 fastest."""
    return _blocks(case["m"], (case["n3"], case["n2"], case["n1"]), case["delta"], _gen(seed))


def _field_lines(case, axis):
    n1, n2, n3 = case["n1"], case["n2"], case["n3"]
    e = n1 * n2 * n3
    return {"x": pbt.Lines(n2, n3, n1, n1 * n2, 1, e), "y": pbt.Lines(n1, n3, 1, n1 * n2, n1, e),
            "z": pbt.Lines(n1, n2, 1, n1, n1 * n2, e)}[axis]


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind, prec = case["kind"], case.get("precision")
    st = {"case": case}
    if kind in ("solve", "grad"):
        A, B, C, d = _solve_inputs(case, seed)
        st["abc"] = [x.reshape(-1) for x in (A, B, C)]
        st["d"] = d.reshape(-1)
        st["plan"] = pbt.BtdmaGpuPlan().create(case["m"], case["nsys"], case["nrow"], case["nseg"], precision=prec,
                                               cyclic=case.get("cyclic", False))
        if kind == "grad":
            st["w"] = _uniform(st["d"].shape, _gen(seed + 1000003))
            for x in st["abc"] + [st["d"]]:
                x.requires_grad_(True)
        else:
            st["x"] = torch.empty_like(st["d"])
    elif kind == "batch":
        m, n, user, _ = _batch_inputs(case, seed)
        plan = pbatch.BatchPlan(m.numpy(), n.numpy(), prec,
                                {"seg_len": {k: case["seg_len"] for k in range(1, 11)}, "warps_per_cta": 4})
        st["plan"], st["packed"] = plan, plan.pack(*user)
        st["d"] = st["packed"][3].clone()
        st["x"] = torch.empty_like(user[3])
    elif kind == "heat":
        h = case["halo"]
        st["field"] = _heat_field(case, seed)
        st["out"] = st["field"].clone()
        st["rhs"], st["x"] = (f[h:-h, h:-h, h:-h] for f in (st["field"], st["out"]))
        st["lines"] = [_heat_lines(case, st["x"], axis) for axis in range(3)]
        st["matrix"] = pshared.SharedMatrix(2, case["n"] // 2, *pshared.heat3d_blocks(case["n"] // 2, case["sigma"]),
                                            precision=prec)
    else:
        A, B, C, d = _field_inputs(case, seed)
        st["abc"], st["d"], st["x"] = [A, B, C], d, torch.empty_like(d)
        st["steps"], plans = [], {}
        rows = {"x": case["n1"], "y": case["n2"], "z": case["n3"]}
        total = case["n1"] * case["n2"] * case["n3"]
        for axis in case["sweeps"]:
            if rows[axis] not in plans:
                plans[rows[axis]] = pbt.BtdmaGpuPlan().create(case["m"], total // rows[axis], rows[axis], 1,
                                                              precision=prec)
            st["steps"].append((plans[rows[axis]], _field_lines(case, axis)))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        x = st["x"].copy_(st["d"])
        f = pbt.solve_cyclic if case["cyclic"] else pbt.solve_noncyclic
        f(st["plan"], *st["abc"], x, case["m"], case["nsys"], case["nrow"])
        return x
    if kind == "grad":
        leaves = st["abc"] + [st["d"]]
        x = pbt.BlockTridiagonalSolve.apply(*leaves, st["plan"])
        return [x.detach()] + list(torch.autograd.grad(x, leaves, st["w"]))
    if kind == "batch":
        p = st["packed"]
        p[3].copy_(st["d"])
        st["plan"].solve(*p)
        return st["plan"].unpack(p[3], st["x"])
    if kind == "heat":
        st["matrix"].solve(st["rhs"], st["x"], st["lines"][0])
        st["matrix"].solve(st["x"], st["x"], st["lines"][1])
        st["matrix"].solve(st["x"], st["x"], st["lines"][2])
        return st["x"]
    x = st["x"].copy_(st["d"])
    for plan, lines in st["steps"]:
        pbt.solve_noncyclic_lines(plan, *st["abc"], x, lines)
    return x


def work(case):
    kind = case["kind"]

    def per_row(m):
        return 8.0 * (3 * m * m + 2 * m), 14.0 / 3.0 * m ** 3 + 8.0 * m * m

    if kind == "solve":
        b, f = per_row(case["m"])
        rows = case["nsys"] * case["nrow"]
        return {"bytes": b * rows, "flops": f * rows}
    if kind == "grad":  # forward; then A, B, C, x, dL/dx read and the four gradients written
        m, rows = case["m"], case["nsys"] * case["nrow"]
        b, f = per_row(m)
        return {"bytes": (b + 8.0 * (6 * m * m + 3 * m)) * rows, "flops": (2 * f + 3 * m * m) * rows}
    if kind == "batch":
        m, n = _uneven_shapes(case)
        t = [(per_row(mm), int(n[m == mm].sum())) for mm in range(case["mmin"], case["mmax"] + 1)]
        return {"bytes": sum(b * r for (b, _), r in t), "flops": sum(f * r for (_, f), r in t)}
    points = case["n"] ** 3 if kind == "heat" else case["n1"] * case["n2"] * case["n3"]
    if kind == "heat":  # three sweeps: rhs read, x written; 3*m*m multiply-adds a row of m = 2 points
        return {"bytes": 3 * 16.0 * points, "flops": 3 * 12.0 * points}
    b, f = per_row(case["m"])
    return {"bytes": len(case["sweeps"]) * b * points, "flops": len(case["sweeps"]) * f * points}


# ---------------------------------------------------------------------------
# The same results in 64 bits: block cyclic reduction with torch.linalg.
# ---------------------------------------------------------------------------
def _reduce(A, B, C, d):
    """x of the non-cyclic systems along dim 0: A, B, C [N, S, m, m], d [N, S,
    m, k]; A[0] and C[-1] must be zero."""
    N, m = B.shape[0], B.shape[-1]
    if N == 1:
        return torch.linalg.solve(B, d)
    odd = torch.linalg.solve(B[1::2], torch.cat([A[1::2], C[1::2], d[1::2]], dim=-1))
    va, vc, vd = odd[..., :m], odd[..., m:2 * m], odd[..., 2 * m:]
    b, r = B[0::2].clone(), d[0::2].clone()
    a, c = torch.zeros_like(b), torch.zeros_like(b)
    left, right = A[0::2][1:], C[0::2][:va.shape[0]]  # even rows q = 2, 4, ... and those with a row q + 1
    k, h = left.shape[0], right.shape[0]
    b[1:] -= left @ vc[:k]
    r[1:] -= left @ vd[:k]
    a[1:] = -(left @ va[:k])
    b[:h] -= right @ va
    r[:h] -= right @ vd
    c[:h] = -(right @ vc)
    even = _reduce(a, b, c, r)
    x = torch.empty_like(d)
    x[0::2] = even
    o = vd - va @ even[:h]
    n = min(h, even.shape[0] - 1)
    o[:n] -= vc[:n] @ even[1:n + 1]
    x[1::2] = o
    return x


def _thomas(A, B, C, d, chunk=1 << 21):
    """_reduce over chunks of systems; A, B, C [j, i, N, S], d [i, N, S]."""
    m, N, S = d.shape
    x = torch.empty_like(d)
    step = max(1, chunk // N)
    for s in range(0, S, step):
        a, b, c = (t[..., s:s + step].permute(2, 3, 1, 0).contiguous() for t in (A, B, C))
        a[0], c[-1] = 0.0, 0.0
        x[..., s:s + step] = _reduce(a, b, c, d[..., s:s + step].permute(1, 2, 0).unsqueeze(-1).contiguous())[
            ..., 0].permute(2, 0, 1)
    return x


def _periodic(A, B, C, d, chunk=1 << 21):
    """Row 0 as the anchor: rows 1.. solved for d and for the columns that
    couple to x_0."""
    m, N, S = d.shape
    x = torch.empty_like(d)
    step = max(1, chunk // N)
    for s in range(0, S, step):
        a, b, c = (t[..., s:s + step].permute(2, 3, 1, 0).contiguous() for t in (A, B, C))
        r = d[..., s:s + step].permute(1, 2, 0).unsqueeze(-1)
        rhs = torch.zeros((N - 1,) + b.shape[1:-1] + (m + 1,), dtype=F64, device=d.device)
        rhs[..., :1] = r[1:]
        rhs[0, ..., 1:] -= a[1]
        rhs[-1, ..., 1:] -= c[-1]
        a1, c1 = a[1:].clone(), c[1:].clone()
        a1[0], c1[-1] = 0.0, 0.0
        y = _reduce(a1, b[1:], c1, rhs)
        x0 = torch.linalg.solve(b[0] + a[0] @ y[-1, ..., 1:] + c[0] @ y[0, ..., 1:],
                                r[0] - a[0] @ y[-1, ..., :1] - c[0] @ y[0, ..., :1])
        out = torch.cat([x0.unsqueeze(0), y[..., :1] + y[..., 1:] @ x0], dim=0)
        x[..., s:s + step] = out[..., 0].permute(2, 0, 1)
    return x


def _exact_grad(case, seed):
    A, B, C, d = _solve_inputs(case, seed)
    x = _thomas(A, B, C, d)
    w = _uniform((d.numel(),), _gen(seed + 1000003)).reshape(d.shape)
    at, ct = torch.zeros_like(A), torch.zeros_like(C)
    at[:, :, 1:] = C[:, :, :-1].transpose(0, 1)
    ct[:, :, :-1] = A[:, :, 1:].transpose(0, 1)
    lam = _thomas(at, B.transpose(0, 1).contiguous(), ct, w)
    xm, xp = torch.zeros_like(x), torch.zeros_like(x)
    xm[:, 1:], xp[:, :-1] = x[:, :-1], x[:, 1:]
    grads = [-(v.unsqueeze(1) * lam.unsqueeze(0)) for v in (xm, x, xp)]  # [j, i, N, S]
    return [v.reshape(-1) for v in [x] + grads + [lam]]


def _exact_batch(case, seed):
    _, _, user, groups = _batch_inputs(case, seed)
    out = torch.empty_like(user[3])
    del user
    for mm, (sel, ns, start, A, B, C, d, vec0, nn) in groups.items():
        x = torch.empty_like(d)
        lg = torch.ceil(torch.log2(ns.double())).long()
        for b in lg.unique().tolist():  # systems of similar length, padded with decoupled rows
            pick = (lg == b).nonzero().flatten()
            N = int(ns[pick].max())
            q = torch.arange(N, device=DEV).unsqueeze(1)
            live = q < ns[pick]
            at = torch.where(live, start[pick] + q, 0)
            a, bb, c, r = (t[..., at] * live for t in (A, B, C, d))
            for i in range(mm):
                bb[i, i] += (~live).double()
            y = _thomas(a, bb, c, r)
            x[:, at[live]] = y[:, live]
        for i in range(mm):
            out[vec0 + nn * i] = x[i]
    return out


def _exact_heat(case, seed):
    n, h = case["n"], case["halo"]
    nblk = n // 2
    M = torch.zeros((nblk, 2, nblk, 2), dtype=F64)
    a, b, c = (torch.from_numpy(v).reshape(2, 2, nblk) for v in _heat_blocks(nblk, case["sigma"]))  # [j, i, q]
    for q in range(nblk):
        M[q, :, q] = b[:, :, q].T
        if q > 0:
            M[q, :, q - 1] = a[:, :, q].T
        if q + 1 < nblk:
            M[q, :, q + 1] = c[:, :, q].T
    M = M.reshape(n, n).to(DEV)
    u = _heat_field(case, seed)[h:-h, h:-h, h:-h].contiguous()
    for axis in range(3):
        v = u.movedim(axis, 0).reshape(n, n * n)
        u = torch.linalg.solve(M, v).reshape(n, n, n).movedim(0, axis).contiguous()
    return u


def _heat_blocks(nblk, s):
    """The fourth-order implicit heat operator in blocks of two points, one
    system, element (i, j) of row q at [j, i, q] (flattened)."""
    import numpy as np

    A, B, C = (np.zeros((2, 2, nblk)) for _ in range(3))  # [i, j, q]
    A[0, 0], A[0, 1], A[1, 1] = s, -16 * s, s
    B[0, 0] = B[1, 1] = 1 + 30 * s
    B[0, 1] = B[1, 0] = -16 * s
    C[0, 0], C[1, 0], C[1, 1] = s, -16 * s, s
    A[:, :, 0] = 0
    B[:, :, 0] = [[1 + 20 * s, -6 * s], [-16 * s, 1 + 30 * s]]
    C[:, :, 0] = [[-4 * s, s], [-16 * s, s]]
    A[:, :, -1] = [[s, -16 * s], [s, -4 * s]]
    B[:, :, -1] = [[1 + 30 * s, -16 * s], [-6 * s, 1 + 20 * s]]
    C[:, :, -1] = 0
    return [np.ascontiguousarray(x.transpose(1, 0, 2)).reshape(-1) for x in (A, B, C)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, B, C, d = _solve_inputs(case, seed)
        return (_periodic if case["cyclic"] else _thomas)(A, B, C, d).reshape(-1)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "heat":
        return _exact_heat(case, seed)
    A, B, C, x = _field_inputs(case, seed)
    m, n1, n2, n3 = case["m"], case["n1"], case["n2"], case["n3"]
    dim = {"x": -1, "y": -2, "z": -3}
    for axis in case["sweeps"]:
        t = [v.movedim(dim[axis], -3) for v in (A, B, C, x)]  # [..., rows, outer, inner]
        shape = t[3].shape
        y = _thomas(*(v.reshape(v.shape[:-2] + (-1,)) for v in t))
        x = y.reshape(shape).movedim(-3, dim[axis]).contiguous()
    return x

"""Lines that are regular and well conditioned but not block diagonally dominant,
on plans of several segments and in uneven batches: a singular or nearly singular
last block, a first block whose elimination makes the second singular.  The
two-stage method solves them, so whatever form the library picks has to.

Tolerance: 64 kappa(M) eps, eps = 2^-52 (FP64) or 2^-44 (float-float), kappa in
the infinity norm of the line's dense matrix, which is what a solve that loses
nothing to element growth keeps to."""
import numpy as np
import pytest
import torch

import pascal_btdma_gb300 as pbt
from pascal_btdma_gb300 import batch as B
from pascal_btdma_gb300 import synth
from test_gpu_batch import check, reference
from test_gpu_ring import batch

pytestmark = pytest.mark.gpu
EPS = {"fp64": 2.0 ** -52, "ff": 2.0 ** -44}
KINDS = ["last", "tiny_last", "second", "both"]


def spoil(a, b, c, kind, s):
    """Make the lines s (of [j, i, row, sys] blocks) non-dominant.  Their other
    blocks stay as they are; the blocks that take the diagonal ones' place are
    made regular and well conditioned."""
    m = b.shape[0]
    eye = torch.eye(m, dtype=b.dtype, device=b.device)[:, :, None]

    def firm(x, q, sign=1.0):
        x[:, :, q, s] = 0.5 * x[:, :, q, s] + sign * m * eye

    if kind in ("last", "tiny_last", "both"):
        firm(a, -1)
        firm(c, -2)
        b[:, :, -1, s] *= 0.0 if kind == "last" else 1e-10
    if kind in ("second", "both"):
        for x, q in ((a, 1), (c, 0), (c, 1)):
            firm(x, q)
        firm(a, 2, -1.0)  # B_2 - A_2 B_1^{-1} C_1 stays regular
        A1, B0, C0 = (x[:, :, q, s].permute(2, 1, 0) for x, q in ((a, 1), (b, 0), (c, 0)))  # [sys, i, j]
        b[:, :, 1, s] = (A1 @ torch.linalg.solve(B0, C0)).permute(2, 1, 0)  # B_1 - A_1 B_0^{-1} C_0 = 0


def dense(a, b, c, s):
    """[len(s), N m, N m] of lines s."""
    m, _, N, _ = b.shape
    M = torch.zeros((len(s), N, m, N, m), dtype=b.dtype, device=b.device)
    for q in range(N):
        for x, p in ((a, q - 1), (b, q), (c, q + 1)):
            if 0 <= p < N:
                M[:, q, :, p] = x[:, :, q, s].permute(2, 1, 0)
    return M.reshape(len(s), N * m, N * m)


def vectors(x, s):
    return x[:, :, s].permute(2, 1, 0).reshape(len(s), -1)  # [sys, (row, i)]


def check_lines(M, x, d, prec):
    inv = torch.linalg.inv(M)
    kappa = M.abs().sum(-1).amax(-1) * inv.abs().sum(-1).amax(-1)
    assert float(kappa.max()) < 1e5  # well conditioned
    ref = torch.linalg.solve(M, d.unsqueeze(-1)).squeeze(-1)
    err = (x - ref).abs().amax(-1) / ref.abs().amax(-1)
    assert bool((err <= 64 * kappa * EPS[prec]).all()), (float(err.max()), float(kappa.max()))


# Sizes that are solved from both ends, in one segment with one lane a column,
# through the ring, and in their segments.
SIZES = [(1, 40, 2), (2, 21, 3), (3, 17, 2), (4, 26, 2), (5, 11, 3), (6, 9, 2), (7, 8, 2), (8, 7, 2), (9, 4, 2), (10, 5, 2),
         (5, 8000, 2), (8, 4096, 2), (4, 12000, 2), (4, 12001, 2), (5, 15000, 2), (6, 13000, 2), (3, 15001, 2), (2, 2000, 4)]


@pytest.mark.parametrize("m,nsys,nseg", SIZES)
@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("kind", KINDS)
def test_lines_that_are_not_dominant(cuda, m, nsys, nseg, prec, kind):
    nrow = 4 * nseg + 1
    a, b, c, d = (x.view(m, -1, nrow, nsys) for x in batch(m, nsys, nrow, seed=nsys + m))
    d = d.view(m, nrow, nsys)
    s = torch.unique(torch.tensor([0, nsys // 2, nsys - 1], device=cuda))
    spoil(a, b, c, kind, s)
    rest = torch.randperm(nsys, device=cuda)[:200]
    keep = [x.clone() for x in (a, b, c)]
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, nsys, nrow, nseg, precision=prec)
        for _ in range(2):  # the second solve starts from the first one's workspace
            x = d.clone()
            pbt.solve_noncyclic(plan, a, b, c, x, m, nsys, nrow)
            assert plan.status() == 0
            check_lines(dense(a, b, c, s), vectors(x, s), vectors(d, s), prec)
            check_lines(dense(a, b, c, rest), vectors(x, rest), vectors(d, rest), prec)
        g = torch.rand_like(d)
        lam, grads = g.clone(), [torch.full_like(a, float("nan")) for _ in range(3)]
        pbt.adjoint_noncyclic(plan, a, b, c, x, lam, *grads)
        assert plan.status() == 0
    for t in (s, rest):
        check_lines(dense(a, b, c, t).transpose(1, 2).contiguous(), vectors(lam, t), vectors(g, t), prec)
    assert torch.equal(grads[1], -(x.unsqueeze(1) * lam.unsqueeze(0)))  # [j, i]: -lambda_i x_j
    for u, v in zip(keep, (a, b, c)):
        assert torch.equal(u, v)


@pytest.mark.parametrize("prec", ["fp64", "ff"])
def test_every_line_of_a_batch_that_is_not_dominant(cuda, prec):
    m, nsys, nrow, nseg = 4, 700, 37, 4
    a, b, c, d = (x.view(m, -1, nrow, nsys) for x in batch(m, nsys, nrow, seed=3))
    d = d.view(m, nrow, nsys)
    s = torch.arange(nsys, device=cuda)
    spoil(a, b, c, "last", s)
    x = d.clone()
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, nsys, nrow, nseg, precision=prec)
        pbt.solve_noncyclic(plan, a, b, c, x, m, nsys, nrow)
        assert plan.status() == 0
    check_lines(dense(a, b, c, s), vectors(x, s), vectors(d, s), prec)


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("m,nsys,nseg", [(2, 300, 2), (3, 700, 4), (5, 500, 2), (8, 300, 2)])
@pytest.mark.parametrize("scale", [3e-2, 3e-3, 3e-4, 3e-6])
def test_small_last_blocks_keep_the_parity_bound(cuda, prec, m, nsys, nseg, scale):
    """Element growth of any size, up to the one from which a line is redone and past
    it: the bound of both arithmetics (1e-12) holds, as in the segments."""
    nrow = 9 * nseg
    a, b, c, d = (x.view(m, -1, nrow, nsys) for x in batch(m, nsys, nrow, seed=m))
    d = d.view(m, nrow, nsys)
    s = torch.arange(nsys, device=cuda)
    spoil(a, b, c, "last", s)
    b[:, :, -1] = scale * (a[:, :, -1] + m * torch.eye(m, dtype=a.dtype, device=cuda)[:, :, None])
    x = d.clone()
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, nsys, nrow, nseg, precision=prec)
        pbt.solve_noncyclic(plan, a, b, c, x, m, nsys, nrow)
        assert plan.status() == 0
    M = dense(a, b, c, s)
    kappa = M.abs().sum(-1).amax(-1) * torch.linalg.inv(M).abs().sum(-1).amax(-1)
    assert float(kappa.max()) < 100  # what is lost is lost to growth
    ref = torch.linalg.solve(M, vectors(d, s).unsqueeze(-1)).squeeze(-1)
    err = (vectors(x, s) - ref).abs().amax(-1) / ref.abs().amax(-1)
    assert float(err.max()) <= 1e-12


def columns_batch(seed):
    """Systems of m = 1..6 and N = 16..60, so many of each that the plan solves all
    in one launch by block columns; their last tiles have 1, 31 or 32 lanes."""
    rng = np.random.default_rng(seed)
    m = np.repeat(np.arange(1, 7, dtype=np.int32), [2049, 2079, 2080, 2049, 2079, 2080])
    n = rng.integers(16, 61, size=m.size).astype(np.int32)
    p = rng.permutation(m.size)
    m, n = m[p], n[p]
    return m, n, [synth.dominant(int(m[s]), 1, int(n[s]), seed=seed * 10000 + s, delta=1.5) for s in range(m.size)]


def solve_batch(cuda, m, n, systems, prec, seg):
    user = [np.concatenate([getattr(w, k) for w in systems]) for k in "ABCD"]
    plan = B.BatchPlan(m, n, prec, {"seg_len": {k: seg for k in range(1, 11)}, "warps_per_cta": 4})
    packed = plan.pack(*(torch.from_numpy(x).to(cuda) for x in user))
    d = packed[3].clone()
    out = []
    for _ in range(2):
        packed[3].copy_(d)
        plan.solve(*packed)
        assert plan.status() == (0, 0)
        info = plan.info()  # one launch: several items a tile, no stage of segments
        assert info["stage1_items"] > info["tiles"] and info["stage3_items"] == 0
        out.append(plan.unpack(packed[3]).cpu().numpy())
    plan.destroy()
    assert np.array_equal(*out)
    return out[0]


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("seg", [0, 12, 40])
def test_batch_in_one_launch_matches_oracle(cuda, prec, seg):
    """seg 0: every line from its first row on; 12: from both ends; 40: some of each."""
    m, n, systems = columns_batch(5)
    got = solve_batch(cuda, m, n, systems, prec, seg)
    check(m, n, got, reference(systems), 1e-12)  # the parity bound of both arithmetics


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("kind", ["last", "tiny_last"])
def test_batch_lines_that_are_not_dominant(cuda, prec, kind):
    m, n, systems = columns_batch(6)
    for s in range(0, m.size, 7):
        w, k = systems[s], int(m[s])
        a, b, c = (x.reshape(k, k, int(n[s]), 1) for x in (w.A, w.B, w.C))  # views
        a[:, :, -1, 0] = 0.5 * a[:, :, -1, 0] + k * np.eye(k)
        c[:, :, -2, 0] = 0.5 * c[:, :, -2, 0] + k * np.eye(k)
        b[:, :, -1] *= 0.0 if kind == "last" else 1e-10
    got = solve_batch(cuda, m, n, systems, prec, 12)
    # kappa of these lines is below 1e3 (the dense matrices of the test above)
    check(m, n, got, reference(systems), 64 * 1e3 * EPS[prec])

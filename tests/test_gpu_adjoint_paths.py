"""The adjoint by column lanes, through the ring and by the fused kernel: lambda
equals the solve of the explicitly transposed blocks, the gradient blocks are
the outer products, at the batch sizes that take each path."""
import pytest
import torch

import pascal_btdma_gb300 as pbt
from test_gpu_ring import batch

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the parity bound of both arithmetics


@pytest.mark.parametrize("m,prec,nsys,nseg", [
    (1, "fp64", 17, 1), (2, "ff", 31, 1), (3, "fp64", 9, 1), (5, "ff", 26, 1), (8, "fp64", 7, 1), (10, "ff", 5, 1),  # lanes
    (4, "ff", 27362, 1), (3, "ff", 60002, 1), (4, "fp64", 10642, 1), (6, "fp64", 12000, 1),  # ring
    (4, "fp64", 15000, 2), (5, "ff", 3000, 2),  # one segment for nseg = 2
    (5, "ff", 27500, 1), (2, "fp64", 14001, 1), (4, "fp64", 10641, 1),  # fused (the last: odd, no tensor map)
])
@pytest.mark.parametrize("nrow", [6, 13])
def test_adjoint_paths(cuda, m, prec, nsys, nseg, nrow):
    a, b, c, d = (x.view(m, -1, nrow, nsys) for x in batch(m, nsys, nrow, seed=3 * nsys + m))  # [j, i, row, sys]
    at, ct = torch.zeros_like(a), torch.zeros_like(c)
    at[:, :, 1:] = c[:, :, :-1].transpose(0, 1)
    ct[:, :, :-1] = a[:, :, 1:].transpose(0, 1)
    w = torch.rand_like(d)
    args = (m, nsys, nrow)
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(*args, 1, precision="fp64", direct_loads=True)
        x, lam = d.clone(), w.clone()
        pbt.solve_noncyclic(plan, a, b, c, x, *args)
        pbt.solve_noncyclic(plan, at.contiguous(), b.transpose(0, 1).contiguous(), ct.contiguous(), lam, *args)
    got = [w.clone()] + [torch.full_like(a, float("nan")) for _ in range(3)]
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(*args, nseg, precision=prec)
        pbt.adjoint_noncyclic(plan, a, b, c, x, got[0], *got[1:])
        assert plan.status() == 0
    assert float((got[0] - lam).abs().amax() / lam.abs().amax()) <= TOL
    xm, xp = torch.zeros_like(x), torch.zeros_like(x)
    xm[:, :, 1:], xp[:, :, :-1] = x[:, :, :-1], x[:, :, 1:]
    for g, v in zip(got[1:], (xm, x, xp)):
        assert torch.equal(g, -(v * got[0].transpose(0, 1)))  # [j, i]: -lambda_i x_j

"""The CTA-wide ring (large batches) against direct loads: the same operations,
so the same bits, at partial warps and CTAs, the fewest rows, several waves, in
place, and on strided lines in both orders of their strides."""
import pytest
import torch

import pascal_btdma_gb300 as pbt

pytestmark = pytest.mark.gpu


def batch(m, nsys, nrow, seed):
    """Diagonally dominant A, B, C, d in the reference layout, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a, b, c = (torch.rand((m, m, nrow, nsys), dtype=torch.float64, device="cuda", generator=g) * 2 - 1 for _ in range(3))
    d = torch.rand((m, nrow, nsys), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    s = a.abs().sum(0) + b.abs().sum(0) + c.abs().sum(0)  # [i, row, sys]
    for i in range(m):
        b[i, i] += 1.1 * s[i]
    return [x.reshape(-1) for x in (a, b, c, d)]


@pytest.mark.parametrize("m,prec,nsys", [
    (3, "ff", 60002), (4, "ff", 27392), (4, "ff", 70000),     # 2 lines in the last warp; full warps; partial CTA
    (4, "fp64", 10650), (5, "fp64", 10642), (6, "fp64", 20002), (5, "fp64", 68098), (3, "fp64", 61000),
    (4, "fp64", 20001),  # odd: no tensor map, direct loads
])
@pytest.mark.parametrize("nrow", [2, 3, 17])
@pytest.mark.parametrize("inplace", [False, True])
def test_ring_gives_the_bits_of_direct_loads(cuda, m, prec, nsys, nrow, inplace):
    w = batch(m, nsys, nrow, seed=m * nsys + nrow)
    out = []
    for direct in (False, True):
        x = [t.clone() for t in w]
        with pbt.BtdmaGpuPlan() as plan:
            plan.create(m, nsys, nrow, 1, precision=prec, direct_loads=direct, inplace=inplace)
            pbt.solve_noncyclic(plan, *x, m, nsys, nrow)
            assert plan.status() == 0
        out.append(x)
    for u, v in zip(*out):
        assert torch.equal(u, v)
    assert bool(torch.isfinite(out[0][3]).all())


@pytest.mark.parametrize("m,prec,n1,n2,n3,axis", [
    (4, "ff", 64, 9, 440, "y"), (4, "ff", 416, 70, 6, "z"), (5, "fp64", 96, 7, 113, "y"), (5, "fp64", 160, 67, 5, "z"),
    (4, "fp64", 40, 266, 5, "z"),  # lines not a multiple of 32 along the fast index: direct loads
])
def test_ring_on_strided_lines(cuda, m, prec, n1, n2, n3, axis):
    """The y and z sweeps of a field equal the plain solve of the same systems."""
    rows, outer = (n2, n3) if axis == "y" else (n3, n2)
    plain = batch(m, n1 * outer, rows, seed=n1)
    view = [x.view(-1, rows, outer, n1) for x in plain]
    field = [(v.permute(0, 2, 1, 3) if axis == "y" else v).contiguous() for v in view]  # [e, k, j, i]
    lines = pbt.Lines(n1, n3, 1, n1 * n2, n1, n1 * n2 * n3) if axis == "y" else pbt.Lines(n1, n2, 1, n1, n1 * n2, n1 * n2 * n3)
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, n1 * outer, rows, 1, precision=prec, direct_loads=True)
        pbt.solve_noncyclic(plan, *plain, m, n1 * outer, rows)
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, n1 * outer, rows, 1, precision=prec)
        pbt.solve_noncyclic_lines(plan, *field, lines)
        assert plan.status() == 0
    x = plain[3].view(m, rows, outer, n1)
    assert torch.equal(field[3].view(m, n3, n2, n1), x.permute(0, 2, 1, 3) if axis == "y" else x)

"""One lane per block column (small batches) against one thread per system:
the same operations, so the same bits, at the edges of a warp's groups (32 //
(m + 1) systems a warp), of the rows, in place, on strided lines, and for the
reported outcomes."""
import numpy as np
import pytest
import torch

import pascal_btdma_gb300 as pbt
from pascal_btdma_gb300 import synth
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


def outcome(plan):
    """The zero pivots that a plan reports, or the name of the error."""
    try:
        return plan.status()
    except ArithmeticError as e:
        return type(e).__name__


def both(w, dev, prec, **kw):
    """(A, B, C, D) and outcome of the default plan and of direct loads with
    one thread per system."""
    out = []
    for direct in (False, True):
        a, b, c, d = to_dev(w.arrays, dev)
        with pbt.BtdmaGpuPlan() as plan:
            plan.create(w.m, w.nsys, w.nrow, 1, precision=prec, direct_loads=direct, **kw)
            pbt.solve_noncyclic(plan, a, b, c, d, w.m, w.nsys, w.nrow)
            out.append(([x.cpu().numpy() for x in (a, b, c, d)], outcome(plan)))
    return out


@pytest.mark.parametrize("m", range(1, 11))
@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("warps,extra,nrow,kw", [
    (0, 1, 2, {}), (1, -1, 3, {"inplace": True}), (1, 0, 7, {}), (4, 1, 12, {}), (9, -2, 5, {"threads_per_block": 96}),
])
def test_columns_give_the_bits_of_one_thread(cuda, m, prec, warps, extra, nrow, kw):
    nsys = max(1, 32 // (m + 1) * warps + extra)
    w = synth.dominant(m, nsys, nrow, seed=7 * m + nsys, delta=1.1)
    (x, sx), (y, sy) = both(w, cuda, prec, **kw)
    assert sx == sy == 0
    for u, v in zip(x, y):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("m,per_sm", [(1, 5), (3, 11), (5, 7), (5, 16), (6, 17), (7, 11), (8, 13), (10, 12), (10, 25)])
@pytest.mark.parametrize("prec", ["fp64", "ff"])
def test_columns_with_an_even_share_of_warps_a_cta(cuda, m, per_sm, prec):
    """per_sm warps an SM and one less: CTAs of one SM's share, of a round's
    share past residency (12 warps, 16 up to m = 6), or of four."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for nsys in (32 // (m + 1) * per_sm * sms, 32 // (m + 1) * (per_sm * sms - sms // 2) - 1):
        w = synth.dominant(m, nsys, 3, seed=m, delta=1.1)
        (x, sx), (y, sy) = both(w, cuda, prec)
        assert sx == sy == 0
        for u, v in zip(x, y):
            assert np.array_equal(u, v)


@pytest.mark.parametrize("prec", ["fp64", "ff"])
def test_columns_pivot_and_report_like_one_thread(cuda, prec):
    m, nsys, nrow = 4, 21, 6
    w = synth.dominant(m, nsys, nrow, seed=5)
    B = w.B.reshape(m, m, nrow, nsys)  # [j, i, row, sys]
    B[:, :, :, 3] = B[:, ::-1, :, 3]  # rows reversed: every step pivots
    B[:, 1, 2, 7] = 0.0
    w.A.reshape(m, m, nrow, nsys)[:, 1, 2, 7] = 0.0  # a zero row of R_2 in system 7
    (x, sx), (y, sy) = both(w, cuda, prec)
    # a float-float solution that is not finite is reported first
    assert sx == sy == (1 if prec == "fp64" else "ArithmeticRangeError")
    keep = np.arange(nsys) != 7
    assert np.array_equal(x[3].reshape(-1, nsys)[:, keep], y[3].reshape(-1, nsys)[:, keep])


def test_columns_report_the_range(cuda):
    w = synth.dominant(3, 10, 5, seed=6)
    w.B[11] = 1e-40
    a, b, c, d = to_dev(w.arrays, cuda)
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(3, 10, 5, 1, precision="ff")
        pbt.solve_noncyclic(plan, a, b, c, d, 3, 10, 5)
        with pytest.raises(pbt.ArithmeticRangeError):
            plan.status()


@pytest.mark.parametrize("m,prec", [(2, "ff"), (5, "fp64"), (8, "ff")])
def test_columns_on_strided_lines(cuda, m, prec):
    """Lines along the middle axis of a 3-D field equal the plain solve of the
    same systems."""
    n1, n2, n3 = 5, 9, 4
    w = synth.dominant(m, n1 * n3, n2, seed=8 * m)
    plain = to_dev(w.arrays, cuda)
    field = [x.view(-1, n2, n3, n1).permute(0, 2, 1, 3).contiguous() for x in plain]  # [e, k, j, i]
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, n1 * n3, n2, 1, precision=prec)
        pbt.solve_noncyclic(plan, *plain, m, n1 * n3, n2)
        pbt.solve_noncyclic_lines(plan, *field, pbt.Lines(n1, n3, 1, n1 * n2, n1, n1 * n2 * n3))
        assert plan.status() == 0
    assert torch.equal(field[3], plain[3].view(-1, n2, n3, n1).permute(0, 2, 1, 3))

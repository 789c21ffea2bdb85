"""Which method a plan of several segments takes, seen in the bits of its solution:
the segments where a twisted or one-segment solve measured slower, one segment where
pairs of warps past residency would take turns."""
import pytest
import torch

import pascal_btdma_gb300 as pbt
from test_gpu_ring import batch

pytestmark = pytest.mark.gpu


def solve(w, m, nsys, nrow, nseg, **kw):
    a, b, c, d = (x.clone() for x in w)
    with pbt.BtdmaGpuPlan() as plan:
        plan.create(m, nsys, nrow, nseg, **kw)
        pbt.solve_noncyclic(plan, a, b, c, d, m, nsys, nrow)
        assert plan.status() == 0
    return d


@pytest.mark.parametrize("m,prec,per_sm,nrow,nseg,one", [
    (1, "fp64", 53, 512, 16, False), (1, "ff", 92, 128, 8, False), (4, "ff", 13, 512, 16, False),
    (4, "fp64", 13, 512, 16, False), (3, "fp64", 72, 48, 4, True), (3, "ff", 81, 61, 3, True),
])
def test_method_that_measured_faster(cuda, m, prec, per_sm, nrow, nseg, one):
    nsys = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    w = batch(m, nsys, nrow, seed=m)
    x = solve(w, m, nsys, nrow, nseg, precision=prec)
    y = solve(w, m, nsys, nrow, 1, precision=prec) if one else solve(w, m, nsys, nrow, nseg, precision=prec, reference_method=True)
    assert torch.equal(x, y)

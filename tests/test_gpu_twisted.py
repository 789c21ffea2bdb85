"""Elimination from both ends (plans of nseg > 1 and uneven batches), against
the oracle: group edges of a warp, the fewest rows, odd and even line lengths,
and the outcome of a line reported from both halves."""
import numpy as np
import pytest
import torch

import pascal_btdma_gb300 as pbt
from pascal_btdma_gb300 import batch as B
from pascal_btdma_gb300 import synth
from conftest import per_system_relerr
from gpu_util import gpu_solve, oracle_solve
from test_gpu_batch import check, make_batch, reference

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the parity bound of both arithmetics


@pytest.mark.parametrize("m", range(1, 11))
@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("extra,nrow,nseg", [(0, 6, 2), (1, 7, 2), (-1, 33, 2), (1, 16, 3)])
def test_twisted_matches_oracle(cuda, m, prec, extra, nrow, nseg):
    nsys = max(1, 3 * (32 // (m + 1)) + extra)
    w = synth.dominant(m, nsys, nrow, seed=11 * m + nrow, delta=1.1)
    (A, _, C, D), singular = gpu_solve(w, nseg, precision=prec)
    assert singular == 0
    assert np.array_equal(A, w.A) and np.array_equal(C, w.C)
    assert per_system_relerr(m, nsys, nrow, D, oracle_solve(w, nseg).D) <= TOL


def test_twisted_reports_the_whole_line(cuda):
    """A solution far below 2^-100 where the halves meet is no range failure,
    one that is so small everywhere is; a zero pivot counts once a system."""
    m, nsys, nrow, nseg = 2, 40, 400, 2
    w = synth.dominant(m, nsys, nrow, seed=4, delta=3.0)
    d = w.D.reshape(m, nrow, nsys)
    d[:, 1:-1, :] = 0.0
    (_, _, _, D), singular = gpu_solve(w, nseg, precision="ff")
    x = D.reshape(m, nrow, nsys)
    assert singular == 0 and np.abs(x[:, nrow // 2]).max() < 1e-40 < np.abs(x).max()
    w.D[:] *= 2.0 ** -110
    with pytest.raises(pbt.ArithmeticRangeError):
        gpu_solve(w, nseg, precision="ff")
    w = synth.dominant(m, nsys, nrow, seed=4)
    b = w.B.reshape(m, m, nrow, nsys)
    b[:, :, 0, 5] = 0.0
    b[:, :, -1, 5] = 0.0  # both sides' first rows
    assert gpu_solve(w, nseg)[1] == 1


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("seg", [0, 12])
def test_batch_by_columns_matches_oracle(cuda, prec, seg):
    """Enough short systems for the single launch; block sizes 7, 8 beside it."""
    m, n, systems, user = make_batch(1500, 2, 40, seed=31, mmax=8)
    plan = B.BatchPlan(m, n, prec, {"seg_len": {k: seg for k in range(1, 11)}, "warps_per_cta": 4})
    packed = plan.pack(*(torch.from_numpy(x).to(cuda) for x in user))
    plan.solve(*packed)
    assert plan.status() == (0, 0)
    check(m, n, plan.unpack(packed[3]).cpu().numpy(), reference(systems), TOL)
    plan.destroy()

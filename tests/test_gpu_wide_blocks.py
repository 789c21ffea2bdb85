"""Block sizes 7 to 10: the split row step with its blocks in registers
(single segment, local stage, reduced solve, periodic lines), against the
oracle at the edges of warps and CTAs, of the rows and of the segments."""
import numpy as np
import pytest

from pascal_btdma_gb300 import synth
from conftest import per_system_relerr
from gpu_util import column_subset, gpu_solve, oracle_solve, subset

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the parity bound of both arithmetics


@pytest.mark.parametrize("m", [7, 8, 9, 10])
@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("nsys,nrow,nseg,kw", [
    (1, 2, 1, {}), (33, 7, 1, {"inplace": True}), (65, 9, 3, {}), (31, 16, 4, {"inplace": True}),
    (40, 3, 1, {"cyclic": True}), (33, 13, 2, {"cyclic": True}), (20001, 4, 1, {}), (3001, 6, 2, {}),
])
def test_wide_blocks_match_oracle(cuda, m, prec, nsys, nrow, nseg, kw):
    cyclic = kw.get("cyclic", False)
    w = synth.fill(synth.DOMINANT, m, nsys, nrow, seed=90 * m + nsys, delta=1.2, flags=0 if cyclic else synth.ZERO_ENDS)
    pick = np.unique(np.concatenate([np.arange(min(nsys, 33)), np.arange(max(0, nsys - 40), nsys)]))
    ref = oracle_solve(subset(w, pick), nseg, cyclic=cyclic)
    (_, _, _, D), singular = gpu_solve(w, nseg, precision=prec, **kw)
    assert singular == 0 and np.isfinite(D).all()
    assert per_system_relerr(m, len(pick), nrow, column_subset(m, nsys, nrow, D, pick), ref.D) <= TOL

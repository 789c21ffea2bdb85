"""CTA sizes of the local stage: whatever size the launch picks for its segments
(few systems a segment, sizes that leave a CTA nearly empty, batches that are not
resident at once), the bits are those of 32-thread CTAs."""
import numpy as np
import pytest
import torch

import pascal_btdma_gb300 as pbt
from pascal_btdma_gb300 import synth
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("m,per_sm,extra", [(1, 8, 0), (2, 4, 1), (3, 12, -1), (4, 8, 3), (5, 9, 33), (6, 10, -31),
                                            (5, 20, 5), (8, 8, 1)])
def test_segment_ctas_give_the_same_bits(cuda, m, per_sm, extra, prec):
    """31 segments: the reduced system (62 rows) is solved directly, whose method
    does not depend on the CTA size."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nseg, nsys = 31, per_sm * 32 * sms // 31 + extra
    nrow = 3 * nseg + 1
    w = synth.dominant(m, nsys, nrow, seed=m, delta=1.3)
    out = []
    for tpb in (0, 32):
        a, b, c, d = to_dev(w.arrays, cuda)
        with pbt.BtdmaGpuPlan() as plan:
            plan.create(m, nsys, nrow, nseg, precision=prec, reference_method=True, threads_per_block=tpb)
            pbt.solve_noncyclic(plan, a, b, c, d, m, nsys, nrow)
            assert plan.status() == 0
        out.append(d.cpu().numpy())
    assert np.array_equal(out[0], out[1])

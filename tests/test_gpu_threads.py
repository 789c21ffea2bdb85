"""Plans of one arithmetic and block size but different shared memory a CTA, solved
from several host threads at once, each on its own stream: every launch succeeds and
gives the bits of the same solve alone."""
import threading

import pytest
import torch

import pascal_btdma_gb300 as pbt
from test_gpu_ring import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,prec,sizes,kw", [
    (5, "fp64", (12000, 66000), {}),                                   # the CTA's ring, 3 and 7 warps
    (6, "ff", (27500, 66000), {}),                                     # one thread per system
    (5, "ff", (1000, 5000), {"reference_method": True, "nseg": 31}),   # local stage
    (6, "ff", (15000, 66000), {"cyclic": True}),
])
def test_threads_with_different_shared_memory(cuda, m, prec, sizes, kw):
    kw = dict(kw)
    nseg = kw.pop("nseg", 1)
    nrow = 3 * nseg + 1
    solve = pbt.solve_cyclic if kw.get("cyclic") else pbt.solve_noncyclic
    errors = []

    def work(nsys):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                a, b, c, d = batch(m, nsys, nrow, seed=nsys)
                with pbt.BtdmaGpuPlan() as plan:
                    plan.create(m, nsys, nrow, nseg, precision=prec, **kw)
                    first, x = d.clone(), d.clone()
                    solve(plan, a, b, c, first, m, nsys, nrow, stream=stream)
                    stream.synchronize()
                    start.wait()
                    for k in range(300):
                        x.copy_(d)
                        for _ in range(5):
                            solve(plan, a, b, c, x, m, nsys, nrow, stream=stream)
                        if k % 20 == 0:
                            stream.synchronize()
                    x.copy_(d)
                    solve(plan, a, b, c, x, m, nsys, nrow, stream=stream)
                    assert plan.status() == 0 and torch.equal(x, first)
        except Exception as e:  # reported by the main thread
            errors.append(e)
            start.abort()

    start = threading.Barrier(2 * len(sizes))
    threads = [threading.Thread(target=work, args=(n,)) for n in sizes * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

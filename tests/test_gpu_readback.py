"""A call that fails leaves no copy on its way into the thread's readback buffer.

A join behind long work on one stream fails in one of its allocations; the thread's
next calls read their counts back on another stream.  A copy left behind by the
first call would land in between and change what they read.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def test_failed_join_then_another_stream(cuda):
    import torch
    import hegjoin_b200 as hj
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    dba, dbb = workloads.exp40(700, 3000, 6, np.float32), workloads.exp40(701, 5000, 2, np.float32)
    ta, tb = torch.from_numpy(dba).to(cuda), torch.from_numpy(dbb).to(cuda)
    _, want = oracle.cell_workload(dbb, 2, np.float32(0.01), *[oracle.geometry(dbb, 2, np.float32(0.01))[i] for i in (0, 2)])
    x = torch.rand((4096, 4096), device=cuda)
    first = hj.GridIndex(ta, 6, 0.02)
    hj.join(first, refine="exact").close()
    first.close()
    torch.cuda.synchronize()
    for nth in range(1, 10):
        ia = hj.GridIndex(ta, 6, 0.02, stream=a)
        with torch.cuda.stream(a):
            for _ in range(4 + nth):
                x @ x
        hj.debug_fail_alloc(nth)
        try:
            with pytest.raises(hj.HJError) as e:
                hj.join(ia, refine="exact", stream=a)
            assert e.value.status == hj.HJ_ERR_OOM
        finally:
            hj.debug_fail_alloc(0)
        for _ in range(20):
            ib = hj.GridIndex(tb, 2, 0.01, stream=b)
            assert ib.sort_by_workload() == want
            assert ib.info().n_nonempty_cells > 0
            ib.close()
        ia.close()
        torch.cuda.synchronize()

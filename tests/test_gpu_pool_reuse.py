"""A large join whose buffers the memory pool already holds skips the free-memory query.

The first join fills the pool, the second takes its buffers from it, the third names a
share of the free memory and queries again: the same lists every time.
"""
import numpy as np
import pytest

from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d, dtype", [(2, np.float64), (6, np.float32)])
def test_repeated_large_join(cuda, d, dtype):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(99, 60_000, d, dtype)
    eps = 0.005 if d == 2 else 0.04
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), d, eps)
    want = None
    for opts in ({}, {}, {"mem_fraction": 0.4}):
        res = hj.join(ix, refine="exact", **opts)
        got = (res.total_pairs, *(t.cpu() for t in res.digest()))
        assert res.total_pairs > 20_000_000
        if want is None:
            want = got
        assert got[0] == want[0] and all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
        del res

"""Large joins with results of earlier ones still held, and with a named capacity.

The free-memory query is skipped only where the memory pool holds idle room for the
buffer and the results together: with earlier results alive it has the buffer's alone.
The same lists every time.
"""
import numpy as np
import pytest

from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def test_results_held_and_named_capacity(cuda):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(98, 60_000, 6, np.float32)
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 6, 0.04)
    want, held = None, []
    for opts in ({}, {}, {"result_capacity": 150_000_000}, {"result_capacity": 150_000_000, "keep_keys": True}, {}):
        res = hj.join(ix, refine="exact", **opts)
        got = (res.total_pairs, *(t.cpu() for t in res.digest()))
        assert res.total_pairs > 20_000_000
        want = want or got
        assert got[0] == want[0] and all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
        held.append(res)
    for r in held:
        r.close()
    ix.close()

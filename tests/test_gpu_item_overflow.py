"""Work items whose pairs outgrow the result buffer by themselves.

The capacity is the smallest that a caller can name, and every point is within
epsilon of every other, so an item (512, 256 or 64 queries) has several times the
pairs that the buffer holds: its queries are run in halves.  Against the oracle.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refine,d,n,shards", [("tc_f16", 18, 2000, 1), ("tc_f16", 18, 2000, 2), ("tc_f16", 120, 2000, 1),
                                               ("exact", 18, 4000, 2)])
def test_items_are_cut(cuda, refine, d, n, shards):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(500, n, d, np.float32)
    eps = np.float32(4.0)
    mn, _, nc, _ = oracle.geometry(db, 2, eps)
    off, vals = oracle.join(db, 2, eps, mn, nc)
    assert int(off[-1]) == n * n
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 2, float(eps), [float(x) for x in mn], [int(x) for x in nc])
    lists = [np.zeros(0, np.uint32)] * n
    for r in range(shards):
        res = hj.join(ix, refine=refine, result_capacity=1, shard_count=shards, shard_index=r)
        assert res.stats.n_retries > 0
        o, v = (t.cpu().numpy() for t in res.to_csr(sort_lists=True))
        for q in range(n):
            if o[q + 1] > o[q]:
                assert len(lists[q]) == 0
                lists[q] = v[o[q]:o[q + 1]].astype(np.uint32)
    assert np.array_equal(np.concatenate(lists), vals)


def test_one_query_too_many_is_refused(cuda):
    # as many pairs per query as there are points, more than the least buffer holds
    import torch
    import hegjoin_b200 as hj
    n = 200_000
    db = np.zeros((n, 18), np.float32)
    db[:, 0] = np.linspace(0.0, 1e-3, n, dtype=np.float32)
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 1, 1.0)
    with pytest.raises(hj.HJError) as e:
        hj.join(ix, refine="exact", result_capacity=1, shard_count=n // 64, shard_index=0)
    assert e.value.status == hj.HJ_ERR_OVERFLOW
    ix.close()

"""The warp-per-item exact refine: every dimension it is built for, both of its
forms, and the digests it can give without writing a pair.

A join in one batch evaluates each unordered pair once (symmetric form); the two
shards of a join evaluate both orders.  The grid starts a little less than
epsilon below the data, so some cells have a coordinate of 0 (they visit no cell
but are visited).  One dimension above the kernel's range checks the hand-over
to the block-tiled kernel.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu

SHAPES = [(np.float32, d) for d in range(1, 14)] + [(np.float64, d) for d in range(1, 10)]


def _case(dtype, d, n, target):
    db = workloads.exp40(99, n, d, dtype)
    db[n // 2:n // 2 + 40] = db[0]                      # a crowded spot: lists beyond one item
    k = min(d, 5)
    x = db[:400].astype(np.float64)
    r = np.sqrt(((x[:, None, :] - x[None, :, :]) ** 2).sum(-1))[np.triu_indices(len(x), 1)]
    eps = dtype(np.quantile(r, min(1.0, target / n)))
    mn = (db[:, :k].min(0) - dtype(0.93) * eps).astype(dtype)
    nc = np.ceil((db[:, :k].max(0) + eps - mn) / eps).astype(np.uint32) + 1
    return db, k, eps, mn, nc


def _index(db, k, eps, mn, nc, dev):
    import torch
    import hegjoin_b200 as hj
    return hj.GridIndex(torch.from_numpy(db).to(dev), k, float(eps), [float(x) for x in mn], [int(x) for x in nc])


def _csr(res):
    off, vals = res.to_csr(sort_lists=True)
    return off.cpu().numpy().astype(np.uint64), vals.cpu().numpy().astype(np.uint32)


@pytest.mark.parametrize("dtype,d", SHAPES)
def test_every_dimension_both_forms(cuda, dtype, d):
    import hegjoin_b200 as hj
    db, k, eps, mn, nc = _case(dtype, d, 2501, 40)
    ix = _index(db, k, eps, mn, nc, cuda)
    off, vals = oracle.join(db, k, eps, mn, nc)
    goff, gvals = _csr(hj.join(ix, refine="exact"))
    assert np.array_equal(goff, off) and np.array_equal(gvals, vals)
    parts = [_csr(hj.join(ix, refine="exact", shard_count=2, shard_index=r)) for r in range(2)]
    for q in range(len(db)):
        lists = [v[o[q]:o[q + 1]] for o, v in parts]
        assert not (len(lists[0]) and len(lists[1]))
        assert np.array_equal(np.concatenate(lists), vals[off[q]:off[q + 1]])


@pytest.mark.parametrize("dtype,d", [(np.float32, 1), (np.float32, 2), (np.float64, 2), (np.float32, 3), (np.float64, 5)])
@pytest.mark.parametrize("n", [257, 20_000])
def test_digests_without_pairs(cuda, dtype, d, n):
    import hegjoin_b200 as hj
    db, k, eps, mn, nc = _case(dtype, d, n, 200)
    ix = _index(db, k, eps, mn, nc, cuda)
    off, vals = oracle.join(db, k, eps, mn, nc)
    want = oracle.digest(off, vals)
    stats, got = hj.join_stream(ix, None, refine="exact")
    assert stats.total_pairs == int(off[-1])
    # with a sink the same digests come from the batches
    _, batched = hj.join_stream(ix, lambda *a: None, refine="exact")
    for g, b, w in zip(got, batched, want):
        w = np.asarray(w)
        assert np.array_equal(g.cpu().numpy().view(w.dtype), w)
        assert np.array_equal(b.cpu().numpy().view(w.dtype), w)

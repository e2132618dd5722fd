"""Digests without pairs on crowded cells: the kernel that folds them in registers.

It takes joins of 8 queries per work item on average, which needs some 300,000
points.  Every dimension it is built for, against the digests of the kept join, and
sampled lists against the oracle.  A join of more than 2^34 candidate pairs runs in
several launches, cut by the items' work: here most of it is in the first few.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu

N = 320_000


def _check(db, k, eps, dev, samples):
    import torch
    import hegjoin_b200 as hj
    ix = hj.GridIndex(torch.from_numpy(db).to(dev), k, eps)
    st, dig = hj.join_stream(ix, None, refine="exact")
    assert st.bytes_wanted == 0 and st.total_pairs > 0          # no pair buffer
    q = np.random.default_rng(1).choice(len(db), samples, replace=False).astype(np.uint32)
    counts, vals = oracle.join_lists(db, k, db.dtype.type(eps), q)
    off = np.zeros(len(q) + 1, np.uint64)
    np.cumsum(counts, out=off[1:])
    for g, w in zip(dig, oracle.digest(off, vals)):
        assert np.array_equal(g.cpu().numpy()[q].view(np.asarray(w).dtype), np.asarray(w))
    return st, dig, ix


@pytest.mark.parametrize("dtype,d", [(np.float32, d) for d in range(1, 13)] + [(np.float64, d) for d in range(1, 9)])
def test_every_dimension(cuda, dtype, d):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(1000 + d, N, d, dtype)
    k, eps = (1, 1e-5) if d == 1 else (2, 0.002) if d == 2 else (2, 0.004)
    st, dig, ix = _check(db, k, eps, cuda, 200)
    assert st.n_batches == 1
    res = hj.join(ix, refine="exact")
    assert res.total_pairs == st.total_pairs
    assert all(torch.equal(a, b) for a, b in zip(dig, res.digest()))


def test_several_launches(cuda):
    g = np.random.default_rng(2)
    db = g.uniform(0.0, 1.0, (N + 130_000, 2)).astype(np.float32)
    db[:150_000] = 0.5 + 0.002 * g.uniform(0.0, 1.0, (150_000, 2))     # 2.25e10 pairs in a few cells
    st, dig, ix = _check(db, 2, 0.01, cuda, 100)
    assert ix.info().total_candidates > 1 << 34 and st.n_batches >= 2
    assert int(dig[0].sum(dtype=dig[1].dtype)) == st.total_pairs

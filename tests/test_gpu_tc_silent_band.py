"""Silent points (a cell coordinate of 0) next to one another in the filter's band.

Such a pair belongs to neither point's list, so it is not among the candidates that
bound a small join's buffer, and it must not take room in the band.  All points lie
in one silent cell and within epsilon of each other; one of them is far out in a
dimension that is not indexed, which widens the band until it takes every pair.  One
work item of 511 queries has 130,816 pairs, more than the buffer's 81,920 slots.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [511, 1500])
def test_silent_pairs_take_no_room(cuda, n):
    import torch
    import hegjoin_b200 as hj
    g = np.random.default_rng(400)
    db = g.uniform(0.0, 0.1, (n, 16)).astype(np.float32)
    db[n // 2, 1:] = 1000.0
    eps = np.float32(1.0)
    mn, nc = np.array([-0.5], np.float32), np.array([4], np.uint32)
    off, _ = oracle.join(db, 1, eps, mn, nc)
    assert int(off[-1]) == 0
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 1, 1.0, [-0.5], [4])
    res = hj.join(ix, refine="tc_f16")
    assert res.total_pairs == 0 and res.stats.n_retries == 0 and res.stats.band_pairs == 0


@pytest.mark.parametrize("origin", [-1.5, -0.95])       # all points in cell 1; in the cells 0 (silent) and 1
def test_band_counts_ordered_pairs(cuda, origin):
    # every result pair goes through the recheck, so the band's count is the result's: a pair of
    # two points twice, that of a point with itself and one with a silent point once
    import torch
    import hegjoin_b200 as hj
    n, eps = 511, np.float32(1.0)
    db = np.random.default_rng(401).uniform(0.0, 0.1, (n, 16)).astype(np.float32)
    db[n // 2, 1:] = 1000.0
    off, _ = oracle.join(db, 1, eps, np.array([origin], np.float32), np.array([4], np.uint32))
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 1, 1.0, [origin], [4])
    res = hj.join(ix, refine="tc_f16")
    assert res.stats.n_batches == 1 and res.total_pairs == int(off[-1]) > 0
    assert res.stats.tc_accepts == 0 and res.stats.band_pairs == int(off[-1])

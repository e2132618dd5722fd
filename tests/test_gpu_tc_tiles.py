"""Tensor-core work items of many candidate tiles, over every number of ring stages.

The candidate tiles pass through a ring of shared-memory stages: 8 for d <= 60,
4 up to d = 124, 3 up to 156 and 2 above.  An item of up to 128 query columns
deals its tiles to four MMA issuers, one of up to 256 to two pairs of them, and
only items of several tiles per issuer use a stage more than once.  A list of
few blocks of queries is cut into items of a tile or two, so thousands of lone
points in cells of their own make the list long, beside cells of 100, 250 and
400 points next to a cell of 2,500.  Both ways of finding hits (HJ_TC_DEFER),
in one batch (each unordered pair once) and in several.  Checked against the
oracle.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

CROWDS = {(1, 1): 100, (2, 1): 2500, (1, 2): 250, (4, 1): 90, (5, 2): 400, (4, 3): 1200}


def _points(d):
    """Crowds in cells of side 1 by their first two coordinates, the other d - 2 such that
    about half of the pairs of a crowd lie within 1 of each other."""
    g = np.random.default_rng(100 + d)
    parts = []
    for (x, y), m in CROWDS.items():
        p = g.normal(0.0, np.sqrt(0.33 / (d - 2)), (m, d))
        p[:, 0] = x + g.uniform(0.05, 0.95, m)
        p[:, 1] = y + g.uniform(0.05, 0.95, m)
        parts.append(p)
    lone = np.zeros((2500, d))
    lone[:, 0] = 20.5 + 2 * (np.arange(2500) % 50)
    lone[:, 1] = 1.5 + 2 * (np.arange(2500) // 50)
    db = np.concatenate(parts + [lone]).astype(np.float32)
    return db[g.permutation(len(db))]


@pytest.mark.parametrize("d", [18, 60, 90, 120, 130, 156, 157, 188])
def test_many_tiles_per_item(cuda, monkeypatch, d):
    import torch
    import hegjoin_b200 as hj
    db = _points(d)
    k, eps = 2, np.float32(1.0)
    mn, nc = np.zeros(2, np.float32), np.array([200, 200], np.uint32)
    off, vals = oracle.join(db, k, eps, mn, nc)
    total = int(off[-1])
    assert total > 1_000_000
    for defer in ("0", "1"):
        monkeypatch.setenv("HJ_TC_DEFER", defer)
        ix = hj.GridIndex(torch.from_numpy(db).to(cuda), k, float(eps), [float(x) for x in mn], [int(x) for x in nc])
        for capacity, batches in ((2 * total, 1), (total // 5, 2)):
            res = hj.join(ix, refine="tc_f16", result_capacity=capacity)
            assert min(res.stats.n_batches, 2) == batches
            goff, gvals = res.to_csr(sort_lists=True)
            assert np.array_equal(goff.cpu().numpy().astype(np.uint64), off)
            assert np.array_equal(gvals.cpu().numpy().astype(np.uint32), vals)

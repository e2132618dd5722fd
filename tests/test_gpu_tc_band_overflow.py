"""A batch whose band pairs outgrow the buffer.

When a reservation fails, the band's array keeps slots that were reserved and never
written; the exact recheck must not read them as point positions.  Far points
widen the band until every neighbour pair is rechecked, the estimate is low (its
first sample is a small crowd that does not reach the large one), and the memory
that the buffer reuses holds the ids of a larger dataset.
Checked against the oracle.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu

# cell: points, first coordinate's share of the cell's side
CROWDS = {(1, 1): (100, 0.05, 0.15), (2, 1): (4500, 0.5, 0.95)}


@pytest.mark.parametrize("d", [60, 90])
def test_band_overflow_is_retried(cuda, d):
    import torch
    import hegjoin_b200 as hj
    g = np.random.default_rng(200 + d)
    parts = []
    for (x, y), (m, lo, hi) in CROWDS.items():
        p = g.normal(0.0, np.sqrt(0.33 / (d - 2)), (m, d))
        p[:, 0] = x + g.uniform(lo, hi, m)
        p[:, 1] = y + g.uniform(0.05, 0.95, m)
        parts.append(p)
    lone = np.zeros((2500, d))
    lone[:, 0] = 20.5 + 2 * (np.arange(2500) % 50)
    lone[:, 1] = 1.5 + 2 * (np.arange(2500) // 50)
    db = np.concatenate(parts + [lone]).astype(np.float32)
    k, eps = 2, np.float32(1.0)
    mn, nc = np.zeros(2, np.float32), np.array([200, 200], np.uint32)
    off, vals = oracle.join(db, k, eps, mn, nc)
    big = torch.from_numpy(workloads.exp40(201, 400_000, 2, np.float32)).to(cuda)
    hj.join(hj.GridIndex(big, 2, 0.002), refine="exact").close()
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), k, float(eps), [float(x) for x in mn], [int(x) for x in nc])
    res = hj.join(ix, refine="tc_f16", result_capacity=1000)
    assert res.stats.n_retries > 0 and res.stats.band_pairs > 0
    goff, gvals = res.to_csr(sort_lists=True)
    assert np.array_equal(goff.cpu().numpy().astype(np.uint64), off)
    assert np.array_equal(gvals.cpu().numpy().astype(np.uint32), vals)

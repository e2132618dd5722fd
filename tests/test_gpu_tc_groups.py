"""Tensor-core work items by their groups of 128 query columns.

An item of one group deals its candidate tiles to four accumulators, one of two
groups to two pairs, and one of three or four groups multiplies every tile four
times; each with the epilogue's two ways of finding hits (HJ_TC_DEFER).  One cell
holds every point, so the item sizes are the cell's.  Checked against the oracle.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("defer", ["0", "1"])
@pytest.mark.parametrize("n", [121, 130, 250, 300, 383, 384, 385, 400, 640, 905])
def test_groups(cuda, monkeypatch, n, defer):
    import torch
    import hegjoin_b200 as hj
    monkeypatch.setenv("HJ_TC_DEFER", defer)
    db = workloads.exp40(98, n, 18, np.float32)
    for eps, k in ((np.float32(0.9), 2), (np.float32(0.15), 2)):   # all pairs of one cell; a few cells, few hits
        mn, _, nc, _ = oracle.geometry(db, k, eps)
        ix = hj.GridIndex(torch.from_numpy(db).to(cuda), k, float(eps), [float(x) for x in mn], [int(x) for x in nc])
        goff, gvals = hj.join(ix, refine="tc_f16").to_csr(sort_lists=True)
        off, vals = oracle.join(db, k, eps, mn, nc)
        assert np.array_equal(goff.cpu().numpy().astype(np.uint64), off)
        assert np.array_equal(gvals.cpu().numpy().astype(np.uint32), vals)

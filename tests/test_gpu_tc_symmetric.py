"""The tensor-core filter's symmetric form: each unordered pair evaluated once.

A join whose work items all run in one batch takes, per item, only the cells
after the item's own and the points of its own cell from the item's first query
on, and emits both orders.  Checked against the oracle at the edges of its work
items (query columns in groups of 8, 256 and 512; candidate tiles of 128), over
cells whose coordinate is 0 (they visit no cell but are visited), and against
the split batches of the same join, which evaluate both orders separately.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def _csr(res):
    off, vals = res.to_csr(sort_lists=True)
    return off.cpu().numpy().astype(np.uint64), vals.cpu().numpy().astype(np.uint32)


def _check(db, k, eps, mn, nc, refine, dev, **kw):
    import torch
    import hegjoin_b200 as hj
    ix = hj.GridIndex(torch.from_numpy(db).to(dev), k, float(eps), [float(x) for x in mn], [int(x) for x in nc])
    res = hj.join(ix, refine=refine, **kw)
    off, vals = oracle.join(db, k, eps, mn, nc)
    goff, gvals = _csr(res)
    assert np.array_equal(goff, off) and np.array_equal(gvals, vals)
    return res


@pytest.mark.parametrize("refine", ["tc_f16", "tc_bf16"])
@pytest.mark.parametrize("n", [1, 7, 8, 127, 128, 129, 255, 256, 257, 511, 512, 513, 521, 1025])
def test_one_cell_of_every_edge_size(cuda, n, refine):
    db = workloads.exp40(95, n, 16, np.float32)
    mn, _, nc, _ = oracle.geometry(db, 2, np.float32(0.9))
    _check(db, 2, np.float32(0.9), mn, nc, refine, cuda)              # every pair is a result
    mn, _, nc, _ = oracle.geometry(db, 2, np.float32(0.1))
    _check(db, 2, np.float32(0.1), mn, nc, refine, cuda)              # a few cells


@pytest.mark.parametrize("d", [16, 60, 90, 120, 188])
def test_two_cells_and_wide_operands(cuda, d):
    # two groups of points one cell apart in dimension 0, neither a multiple of 8 long, over
    # the operand sizes with 512 and with 256 query columns per item
    db = workloads.exp40(96, 1003, d, np.float32) * np.float32(0.2)
    db[300:, 0] += np.float32(0.25)
    eps = np.float32(0.24)
    mn, _, nc, _ = oracle.geometry(db, 3, eps)
    _check(db, 3, eps, mn, nc, "tc_f16", cuda)


@pytest.mark.parametrize("refine", ["tc_f16", "tc_bf16"])
def test_silent_cells(cuda, refine):
    # a grid that starts a little less than epsilon below the data's minimum, so that about
    # half of the points have a coordinate of 0 in some dimension
    db = workloads.exp40(97, 20000, 18, np.float32)
    k, eps = 3, np.float32(0.07)
    mn = db[:, :k].min(0) - np.float32(0.9) * eps
    nc = np.ceil((db[:, :k].max(0) + eps - mn) / eps).astype(np.uint32) + 1
    coords = np.trunc((db[:, :k] - mn) / eps)
    silent = (coords == 0).any(1)
    assert 0.3 < silent.mean() < 0.8
    res = _check(db, k, eps, mn, nc, refine, cuda)
    # in several batches (of far more pairs than the warps' partly filled chunks) the items
    # evaluate both orders themselves
    many = _check(db, k, eps, mn, nc, refine, cuda, result_capacity=max(1, res.total_pairs // 6))
    assert many.stats.n_batches > 1

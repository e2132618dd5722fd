"""Sorted neighbour lists of the CSR export, at every list length where its sort changes form.

Groups of identical points far from each other: a group of m points gives m lists
of exactly its m members.  Warps sort lists of up to 32, 64, ... 1,024 values,
blocks the longer ones, in two radix passes for up to 65,536 points and three
above.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 4099]


@pytest.mark.parametrize("alone", [0, 5, 60_000])
def test_lists_of_every_length(cuda, alone):
    import torch
    import hegjoin_b200 as hj
    sizes = np.array(SIZES + [1] * alone)
    if alone == 0:
        sizes = sizes[:-3]                       # no list past a warp's longest
    group = np.repeat(np.arange(len(sizes)), sizes)
    rng = np.random.default_rng(98)
    group = group[rng.permutation(len(group))]
    db = np.stack([(group % 300) / 301.0, (group // 300) / 301.0], 1).astype(np.float64)
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 2, 0.001)
    off, vals = hj.join(ix).to_csr(sort_lists=True)
    off, vals = off.cpu().numpy(), vals.cpu().numpy()
    assert np.array_equal(np.diff(off), sizes[group])
    order = np.argsort(group, kind="stable")     # members of each group, ascending
    first = np.concatenate([[0], np.cumsum(sizes)])
    for g in np.flatnonzero(sizes > 1).tolist() + list(range(len(SIZES), min(len(sizes), len(SIZES) + 5))):
        members = order[first[g]:first[g + 1]]
        for q in (members if len(members) < 300 else members[::97]):
            assert np.array_equal(vals[off[q]:off[q + 1]], members)
    unsorted_off, unsorted = hj.join(ix).to_csr(sort_lists=False)
    assert np.array_equal(unsorted_off.cpu().numpy(), off)
    assert np.array_equal(np.sort(unsorted.cpu().numpy()), np.sort(vals))

"""Index arrays and workload order at the sizes where the sort changes form.

Up to 7,168 points one block sorts everything in shared memory, each of its 32
warps a run of whole 32s; above, tiles of 4,096 keys, 512 per warp.  Few and many
key bits (two and six 8-bit passes for the points).
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,eps", [(2, 0.004), (6, 0.01)])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 1023, 1024, 1025, 4097, 7167, 7168, 7169, 8191, 8192, 8193, 12_801])
def test_index_and_order(cuda, d, eps, n):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(94, n, d, np.float32)
    mn, _, nc, _ = oracle.geometry(db, d, np.float32(eps))
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), d, float(np.float32(eps)), [float(x) for x in mn],
                      [int(x) for x in nc])
    lid, first, last, lookup = oracle.index(db, d, np.float32(eps), mn, nc)
    glid, gfirst, glast, glookup, _ = ix.export()
    assert np.array_equal(glid.cpu().numpy().astype(np.uint64), lid)
    assert np.array_equal(gfirst.cpu().numpy(), first) and np.array_equal(glast.cpu().numpy(), last)
    assert np.array_equal(glookup.cpu().numpy().astype(np.uint32), lookup)
    nb, total = oracle.cell_workload(db, d, np.float32(eps), mn, nc)
    assert ix.sort_by_workload() == total
    sched = ix.workload_export()[0].cpu().numpy()
    order = np.argsort(-nb.astype(np.int64), kind="stable")     # heaviest first, ties by cell
    assert np.array_equal(sched[:, 1], order)
    assert np.array_equal(sched[:, 0], nb[order].astype(np.int32))

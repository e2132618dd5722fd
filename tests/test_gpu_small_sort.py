"""The one-block sort at the sizes whose shared memory ends near 48 KB.

Its dynamic shared memory is 32 KB plus 24 bytes per point (cell ids) or 16 per
cell (workload order), and a little static memory comes on top: 682 points, and
1,023 and 1,024 cells, lie between the two sums.  Each size in a process of its own:
a larger sort before it would have raised the kernel's limit.
"""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import sys
    import numpy as np, torch
    sys.path.insert(0, {root!r})
    import oracle
    import hegjoin_b200 as hj
    n, cells = {n}, {cells}
    # {cells} cells in a row of a 2-D grid, the points dealt to them in turn
    i = np.arange(n)
    db = np.stack([(i % cells) * 0.25 + 0.125, np.full(n, 0.5)], 1).astype(np.float32)
    mn, nc = [0.0, 0.0], [4096, 8]
    ix = hj.GridIndex(torch.from_numpy(db).cuda(), 2, 0.25, mn, nc)
    a = (db, 2, np.float32(0.25), np.zeros(2, np.float32), np.array(nc, np.uint32))
    nb, total = oracle.cell_workload(*a)
    assert len(nb) == cells and ix.sort_by_workload() == total
    lid, first, last, lookup = oracle.index(*a)
    glid, gfirst, glast, glookup, _ = ix.export()
    assert np.array_equal(glid.cpu().numpy().astype(np.uint64), lid)
    assert np.array_equal(glookup.cpu().numpy().astype(np.uint32), lookup)
    order = np.argsort(-nb.astype(np.int64), kind="stable")
    sched = ix.workload_export()[0].cpu().numpy()
    assert np.array_equal(sched[:, 1], order) and np.array_equal(sched[:, 0], nb[order].astype(np.int32))
    print("OK")
""")


@pytest.mark.parametrize("n,cells", [(681, 100), (682, 100), (683, 100), (8000, 1022), (8000, 1023), (8000, 1024),
                                     (8000, 1025)])
def test_sizes_near_the_limit(cuda, n, cells):
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, n=n, cells=cells)], capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0 and "OK" in p.stdout, p.stderr[-2000:]

"""Index builds after the process has reset its device.

cudaDeviceReset ends the process's context, and with it the pinned buffer that
readbacks of an earlier call went through and the shared-memory limits that were
raised for its kernels.  The next call works in a new context.  In a process of its
own, through the C interface; up to 7,168 points the sort needs a raised limit.
"""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import ctypes, sys
    import numpy as np
    sys.path.insert(0, {root!r})
    import oracle
    import hegjoin_b200 as hj
    from hegjoin_b200 import workloads
    from cuda.bindings import runtime as rt
    for n in (20000, 30000, 3000, 7000):
        db = workloads.exp40(800, n, 2, np.float32)
        mn, _, nc, _ = oracle.geometry(db, 2, np.float32(0.01))
        cells = len(oracle.index(db, 2, np.float32(0.01), mn, nc)[0])
        e, p = rt.cudaMalloc(db.nbytes)
        assert int(e) == 0, e
        assert int(rt.cudaMemcpy(p, db.ctypes.data, db.nbytes, rt.cudaMemcpyKind.cudaMemcpyHostToDevice)[0]) == 0
        h = ctypes.c_void_p()
        hj.check(hj.lib.hj_index_create(p, n, 2, 2, hj.HJ_F32, 0.01, None, None, None, ctypes.byref(h)))
        info = hj.IndexInfo()
        hj.check(hj.lib.hj_index_get_info(h, ctypes.byref(info)))
        assert info.n_nonempty_cells == cells, (info.n_nonempty_cells, cells)
        hj.check(hj.lib.hj_index_destroy(h))
        assert int(rt.cudaDeviceReset()[0]) == 0
    print("OK")
""")


def test_index_after_device_reset(cuda):
    pytest.importorskip("cuda.bindings.runtime")
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "OK" in p.stdout, p.stderr[-2000:]

"""One index joined by several threads at once, each on a stream of its own.

With its workload order made (and, for the filter, its operand forms by an earlier
join), an index is only read by joins.  Coordinates with an offset: in FP32 the
grid's first cells then get a coordinate of 0, whose points the joins have to
know.  Every index is new, so each round has a first join on either stream.
Checked against the oracle.
"""
import threading

import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def _join_together(ix, streams, options, off, vals):
    import torch
    import hegjoin_b200 as hj
    start = threading.Barrier(len(streams))
    got, errors = [None] * len(streams), []

    def work(i):
        try:
            start.wait()
            for _ in range(3):
                with torch.cuda.stream(streams[i]):
                    o, v = hj.join(ix, **options[i]).to_csr(sort_lists=True)
                    got[i] = (o.cpu().numpy().astype(np.uint64), v.cpu().numpy().astype(np.uint32))
                assert np.array_equal(got[i][0], off) and np.array_equal(got[i][1], vals)
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(streams))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("d,k,eps,offset", [(6, 6, 0.03, 100.0), (2, 2, 0.004, 100.0)])
def test_exact_joins_of_one_index(cuda, d, k, eps, offset):
    import torch
    import hegjoin_b200 as hj
    streams = [torch.cuda.Stream() for _ in range(4)]
    for seed in range(6):
        db = (workloads.exp40(300 + seed, 9000, d, np.float32) + np.float32(offset)).astype(np.float32)
        mn, _, nc, _ = oracle.geometry(db, k, np.float32(eps))
        coords = ((db[:, :k] - mn) / np.float32(eps)).astype(np.int64)
        assert (coords == 0).any()
        off, vals = oracle.join(db, k, np.float32(eps), mn, nc)
        ix = hj.GridIndex(torch.from_numpy(db).to(cuda), k, eps)
        ix.sort_by_workload()
        torch.cuda.synchronize()
        _join_together(ix, streams, [{"refine": "exact"}] * 4, off, vals)


def test_filter_joins_of_one_index(cuda):
    # operand forms made by the tile probe: the joins count their samples in the filter's sparse
    # form and then run the dense one, each on its own account
    import torch
    import hegjoin_b200 as hj
    streams = [torch.cuda.Stream() for _ in range(4)]
    db = workloads.exp40(310, 6000, 18, np.float32)
    eps = np.float32(0.07)
    off, vals = oracle.join(db, 6, eps)
    for _ in range(8):
        ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 6, float(eps))
        ix.sort_by_workload()
        hj.probe_tc_tile(ix, "tc_f16", 0, 0)
        torch.cuda.synchronize()
        _join_together(ix, streams, [{"refine": "tc_f16"}] * 4, off, vals)

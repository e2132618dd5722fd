"""The exact refine's two forms in whole joins, on both sides of the rule between them.

A join in one batch evaluates each unordered pair once where that saves enough
distances per result pair, and both orders where results are dense (2-D and 3-D
here).  A capacity keeps the joins from being sized by their candidates, which
leaves the choice aside.  Lists, kept keys and a sink's batches against the oracle.
"""
import numpy as np
import pytest

import oracle
from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d,eps", [(2, 0.004), (3, 0.01), (4, 0.012), (5, 0.014), (7, 0.02)])
def test_lists_keys_and_batches(cuda, dtype, d, eps):
    import torch
    import hegjoin_b200 as hj
    n = 12_000
    db = workloads.exp40(600, n, d, dtype) + dtype(1)      # FP32: some cells have a coordinate of 0
    eps = float(dtype(eps))
    off, vals = oracle.join(db, d, dtype(eps))
    total = int(off[-1])
    counts = np.diff(off.astype(np.int64))
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), d, eps)
    res = hj.join(ix, refine="exact", result_capacity=4 * total, keep_keys=True)
    assert res.stats.n_batches == 1 and res.total_pairs == total
    goff, gvals = res.to_csr(sort_lists=True)
    assert np.array_equal(goff.cpu().numpy().astype(np.uint64), off)
    assert np.array_equal(gvals.cpu().numpy().astype(np.uint32), vals)
    (_, kp, m), = res.batches()
    keys = hj.device_view(kp, (m,), np.int32).cpu().numpy()
    assert np.array_equal(keys, np.repeat(np.arange(n, dtype=np.int32), counts))
    plain = hj.join(ix, refine="exact", result_capacity=4 * total)
    goff, gvals = plain.to_csr(sort_lists=True)
    assert np.array_equal(goff.cpu().numpy().astype(np.uint64), off)
    assert np.array_equal(gvals.cpu().numpy().astype(np.uint32), vals)
    got = {}

    def sink(batch, count, kp, vp, stream):
        got[batch] = (hj.device_view(kp, (count,), np.int32).clone(), hj.device_view(vp, (count,), np.int32).clone())

    st, dig = hj.join_stream(ix, sink, refine="exact", result_capacity=4 * total)
    torch.cuda.synchronize()
    assert st.total_pairs == total and len(got) == 1
    k, v = (x.cpu().numpy() for x in got[0])
    assert np.array_equal(k, keys)
    order = np.lexsort((v, k))
    assert np.array_equal(v[order].astype(np.uint32), vals)
    for g, w in zip(dig, oracle.digest(off, vals)):
        assert np.array_equal(g.cpu().numpy().view(np.asarray(w).dtype), np.asarray(w))

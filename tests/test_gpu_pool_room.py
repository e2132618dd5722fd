"""Large joins with results of earlier ones still held, and with a named capacity.

The free-memory query is skipped where the memory pool holds the join's buffer idle.
Where the results then find no memory, the join sizes its buffer by the free memory
after all.  The same lists every time.
"""
import numpy as np
import pytest

from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def test_results_held_and_named_capacity(cuda):
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(98, 60_000, 6, np.float32)
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 6, 0.04)
    want, held = None, []
    for opts in ({}, {}, {"result_capacity": 150_000_000}, {"result_capacity": 150_000_000, "keep_keys": True}, {}):
        res = hj.join(ix, refine="exact", **opts)
        got = (res.total_pairs, *(t.cpu() for t in res.digest()))
        assert res.total_pairs > 20_000_000
        want = want or got
        assert got[0] == want[0] and all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
        held.append(res)
    for r in held:
        r.close()
    ix.close()


def _refusals(ix, want, **opts):
    """Allocations of the join that end it when they fail once."""
    import torch
    import hegjoin_b200 as hj
    hj.join(ix, refine="exact", **opts).close()
    refused = 0
    for nth in range(1, 60):
        torch.cuda.synchronize()
        base = hj.debug_pool_used()
        hj.debug_fail_alloc(nth)
        try:
            res = hj.join(ix, refine="exact", **opts)
        except hj.HJError as e:
            assert e.status == hj.HJ_ERR_OOM
            refused += 1
            torch.cuda.synchronize()
            assert hj.debug_pool_used() == base
            continue
        finally:
            hj.debug_fail_alloc(0)
        got = (res.total_pairs, *(t.cpu() for t in res.digest()))
        assert got[0] == want[0] and all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
        res.close()
    return refused


def test_an_allocation_that_fails_beside_an_idle_pool(cuda):
    # with the buffer's memory idle in the pool, a failure of the buffer's allocation or of a later
    # one (counters, values, batch pointers) does not end the join
    import torch
    import hegjoin_b200 as hj
    db = workloads.exp40(97, 60_000, 6, np.float32)
    ix = hj.GridIndex(torch.from_numpy(db).to(cuda), 6, 0.04)
    first = hj.join(ix, refine="exact")
    want = (first.total_pairs, *(t.cpu() for t in first.digest()))
    first.close()
    assert _refusals(ix, want) <= _refusals(ix, want, mem_fraction=0.5) - 4
    ix.close()

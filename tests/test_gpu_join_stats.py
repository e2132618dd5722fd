"""What a join's statistics say where it makes no estimate, and of a shard's share."""
import numpy as np
import pytest

from hegjoin_b200 import workloads

pytestmark = pytest.mark.gpu


def _index(cuda, n, d, eps):
    import torch
    import hegjoin_b200 as hj
    return hj.GridIndex(torch.from_numpy(workloads.exp40(900, n, d, np.float32)).to(cuda), min(d, 6), eps)


@pytest.mark.parametrize("n,d,eps,refine", [(2000, 2, 0.005, "exact"), (1000, 18, 0.05, "tc_f16")])
def test_small_joins(cuda, n, d, eps, refine):
    import hegjoin_b200 as hj
    ix = _index(cuda, n, d, eps)
    whole = hj.join(ix, refine=refine)
    assert whole.stats.estimated_pairs == whole.total_pairs > 0
    parts = [hj.join(ix, refine=refine, shard_count=2, shard_index=r) for r in range(2)]
    assert sum(p.total_pairs for p in parts) == whole.total_pairs
    for p in parts:
        assert p.stats.estimated_pairs == p.total_pairs
        assert p.stats.bytes_wanted < whole.stats.bytes_wanted


def test_digests_alone(cuda):
    import hegjoin_b200 as hj
    ix = _index(cuda, 320_000, 2, 0.002)      # enough points per work item for the digest kernel
    st, _ = hj.join_stream(ix, None, refine="exact")
    assert st.estimated_pairs == st.total_pairs > 0 and st.bytes_wanted == 0

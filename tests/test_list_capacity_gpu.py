"""Batches so large that the candidate lists take their smaller capacity: the
same rows as from calls under that line, bit for bit."""
import pytest
import torch

from mlxlearn_b200.index import NeighborIndex

pytestmark = pytest.mark.gpu


# four lists of 512 entries a query pass 32 GB above 2,097,152 queries
@pytest.mark.parametrize("d,k", [(20, 17), (8, 5)])
def test_large_batch_equals_its_parts(d, k):
    g = torch.Generator(device="cuda").manual_seed(d)
    X = torch.randn(9_000, d, generator=g, device="cuda")
    X[100:140] = X[:40]  # duplicates
    Q = torch.randn(2_200_000, d, generator=g, device="cuda")
    index = NeighborIndex.from_device(X)
    dist, idx = index.query_device(Q, k)
    for a, b in ((0, 100_000), (2_100_000, 2_200_000)):
        part_dist, part_idx = index.query_device(Q[a:b], k)
        assert torch.equal(idx[a:b], part_idx)
        assert torch.equal(dist[a:b], part_dist)

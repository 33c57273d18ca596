"""Index build on the device: rows grouped by pivot (a stable counting sort),
buffers from the pool, inputs produced on the caller's stream."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import NeighborIndex, build_index

pytestmark = pytest.mark.gpu


# 8192: the smallest grouped index; tiles of 512 rows with remainders; even
# groups, and nearly all rows in one
@pytest.mark.parametrize("n", [8192, 8193, 8704, 20000])
@pytest.mark.parametrize("skew", [False, True])
def test_grouped_self_query(n, skew):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 24)).astype(np.float32)
    if skew:
        X[rng.permutation(n)[: n - n // 50]] *= np.float32(1e-3)
    index = build_index(X)
    dist, idx = index.query(X, 3, exclude_self=True)
    rows = rng.choice(n, 500, replace=False)
    ed, ei = oracle.knn(X, X[rows], 4)  # the row itself first (distinct rows)
    assert np.array_equal(ei[:, 0], rows)
    assert np.array_equal(idx[rows], ei[:, 1:])
    assert np.array_equal(dist[rows], ed[:, 1:])


def test_rows_produced_on_the_callers_stream():
    import torch

    # the copy into the index waits for the work that produces its rows
    for side in (None, torch.cuda.Stream()):
        with torch.cuda.stream(side):
            a = torch.randn(4096, 4096, device="cuda")
            X = torch.zeros(9000, 32, device="cuda")
            for _ in range(20):
                a = (a @ a).clamp_(-1, 1)
            X += torch.arange(9000, device="cuda")[:, None] + 0 * a[0, 0]
            index = NeighborIndex.from_device(X)
            assert np.array_equal(index.training_data, X.cpu().numpy())


def test_many_short_lived_indexes():
    rng = np.random.default_rng(3)
    for i in range(12):
        X = rng.standard_normal((2048 + 700 * i, 20)).astype(np.float32)
        index = build_index(X)
        dist, idx = index.query(X[:50], 4)
        ed, ei = oracle.knn(X, X[:50], 4)
        assert np.array_equal(idx, ei)
        assert np.array_equal(dist, ed)
        index.close()

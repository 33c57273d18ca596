"""Batches with a seeding pass: problems just below and above its smallest size,
ordered rows (an unrepresentative sample) and ties, bit for bit against the
oracle."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.batch import KnnBatch
from mlxlearn_b200.index import NeighborIndex

pytestmark = pytest.mark.gpu


# eight tiles of 256 rows: 1,792 rows have seven, 1,793 the eighth
@pytest.mark.parametrize("order", ["random", "near_last", "near_first"])
def test_seeded_batch(order):
    import torch

    rng = np.random.default_rng(11)
    data, problems = [], []
    for n, m, d, k in ((1792, 130, 16, 10), (1793, 129, 16, 10), (5000, 300, 40, 50),
                       (9000, 77, 64, 64), (4097, 128, 21, 1), (20000, 260, 100, 17),
                       (3000, 1, 300, 16)):
        X = rng.standard_normal((n, d)).astype(np.float32)
        X[rng.choice(n, n // 50, replace=False)] = X[rng.integers(0, n, n // 50)]
        if order != "random":
            by_norm = np.argsort((X * X).sum(1))
            X = X[by_norm if order == "near_first" else by_norm[::-1]].copy()
        Q = (0.5 * rng.standard_normal((m, d))).astype(np.float32)
        data.append((X, Q, k))
        problems.append((NeighborIndex.from_device(torch.from_numpy(X).cuda()),
                         torch.from_numpy(Q).cuda(), k))
    batch = KnnBatch(problems)
    for _ in range(2):  # a replay starts from cleared words
        for (dist, idx), (X, Q, k) in zip(batch(), data):
            ed, ei = oracle.knn(X, Q, k)
            assert np.array_equal(idx.cpu().numpy(), ei)
            assert np.array_equal(dist.cpu().numpy(), ed)

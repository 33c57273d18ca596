"""Segments of narrow rows (d <= 8): the scan skips rows by a centred bound and
must still give exactly the oracle's answer, wherever the data lies."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _check(Qs, Xs, k, exclude_self=False):
    import torch

    from mlxlearn_b200.autograd import knn_segments

    Q = torch.from_numpy(np.concatenate(Qs)).cuda()
    X = torch.from_numpy(np.concatenate(Xs)).cuda()
    dist, idx = knn_segments(Q, X, [len(q) for q in Qs], [len(x) for x in Xs], k,
                             exclude_self=exclude_self)
    ref = [oracle.knn(x, q, k, exclude_self=exclude_self) for q, x in zip(Qs, Xs)]
    assert np.array_equal(idx.cpu().numpy(), np.concatenate([i for _, i in ref]))
    # the float32 output holds the canonical distance rounded
    assert np.array_equal(dist.cpu().numpy(),
                          np.concatenate([d for d, _ in ref]).astype(np.float32))


# tiles of 512 rows read eight at a time: sizes around both, and the smallest
@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("k", [1, 5, 13, 29])
def test_sizes(d, k):
    rng = np.random.default_rng(31 * d + k)
    sizes = [n for n in (1, 2, 7, 8, 9, 31, 33, 511, 512, 513, 1024, 1031) if n >= k]
    Xs = [rng.standard_normal((n, d)).astype(np.float32) for n in sizes]
    Qs = [rng.standard_normal((int(rng.integers(1, 300)), d)).astype(np.float32) for _ in sizes]
    _check(Qs, Xs, k)


# far from the origin, two distant clumps of close points, spread over 2^40
@pytest.mark.parametrize("kind", ["offset", "clumps", "spread", "lattice"])
@pytest.mark.parametrize("k", [1, 6])
def test_placement(kind, k):
    rng = np.random.default_rng(5)
    if kind == "lattice":  # duplicates: ties everywhere
        X = np.repeat(rng.integers(-2, 3, (250, 3)), 3, axis=0)
    else:
        X = rng.standard_normal((1500, 3))
        if kind == "offset":
            X = 4096.0 + 1e-2 * X
        elif kind == "clumps":
            X = np.where(rng.random((1500, 1)) < 0.5, -500.0, 500.0) + 1e-3 * X
        else:
            X = X * 2.0 ** rng.integers(-20, 21, (1500, 1))
    X = X.astype(np.float32)
    _check([X, X[:40]], [X, X], k)
    _check([X], [X], k, exclude_self=True)


def test_two_queries_a_thread():
    # enough queries for two a thread; ragged last blocks
    rng = np.random.default_rng(9)
    Xs = [rng.standard_normal((int(rng.integers(1, 120)), 3)).astype(np.float32)
          for _ in range(45)]
    Qs = [rng.standard_normal((int(rng.integers(1500, 2400)), 3)).astype(np.float32)
          for _ in range(45)]
    assert sum(map(len, Qs)) > 2 * 128 * 2 * 148
    _check(Qs, Xs, 1)

"""k > 16: the seeded lazy screen and the certify pass over many lists, bit for
bit against the oracle."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


def _rows(n, d, seed, centres):
    rng = np.random.default_rng(seed)
    if not centres:
        return rng.standard_normal((n, d)).astype(np.float32)
    C = np.random.default_rng(1).uniform(-1, 1, (centres, d))
    return (C[rng.integers(0, centres, n)] + 0.1 * rng.standard_normal((n, d))).astype(np.float32)


# 8192 rows: the first grouped (seeded) index, 32 tiles; 17 | 64: the edges of
# the lazy tracker; tight clusters put more rows in the band than a list holds
@pytest.mark.parametrize("n,d,m", [(8191, 40, 2100), (8192, 40, 2100), (20011, 24, 2500)])
@pytest.mark.parametrize("k", [16, 17, 50, 64])
@pytest.mark.parametrize("centres", [0, 8])
def test_large_k(n, d, m, k, centres):
    X, Q = _rows(n, d, n + k, centres), _rows(m, d, 3 * n + k, centres)
    X[100:140] = X[:40]  # duplicates
    dist, idx = build_index(X).query(Q, k)
    ed, ei = oracle.knn(X, Q, k)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


@pytest.mark.parametrize("k", [20, 50])
def test_large_k_self(k):
    X = _rows(9001, 33, k, 100)
    dist, idx = build_index(X).query(X, k, exclude_self=True)
    ed, ei = oracle.knn(X, X, k, exclude_self=True)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


# few queries over many splits: up to 256 short lists a row, walked as one
@pytest.mark.parametrize("m", [1, 3, 129])
@pytest.mark.parametrize("k", [1, 5, 16, 40])
def test_many_lists(m, k):
    X, Q = _rows(30011, 32, 7, 0), _rows(m, 32, 8, 0)
    dist, idx = build_index(X).query(Q, k)
    ed, ei = oracle.knn(X, Q, k)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


# seeding windows spread over the rows: 4 windows of 8 or 9 tiles, one window a
# tile with a ragged end, two tiles a window; 64 is the widest k
@pytest.mark.parametrize("n,m", [(2048, 5), (2049, 300), (20011, 2047), (100003, 1500)])
@pytest.mark.parametrize("d,k", [(5, 17), (20, 64)])
def test_spread_seeding(n, m, d, k):
    X, Q = _rows(n, d, n + m, 0), _rows(m, d, n + d, 50)
    X[100:140] = X[:40]
    Q[:5] = X[:5]
    dist, idx = build_index(X).query(Q, k)
    ed, ei = oracle.knn(X, Q, k)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


def test_spread_seeding_self():
    X = _rows(6001, 12, 3, 30)
    dist, idx = build_index(X).query(X, 30, exclude_self=True)
    ed, ei = oracle.knn(X, X, 30, exclude_self=True)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)

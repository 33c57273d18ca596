"""Rows of few features on the tensor cores: bf16 parts (hi + mid (+ lo)) whose
cross products fill a 64-column block.  Answers are exact, so every comparison
with the oracle is bit for bit."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


def _rows(n, d, seed, offset=0.0, scale=1.0):
    X = (offset + scale * np.random.default_rng(seed).standard_normal((n, d))).astype(np.float32)
    X[n // 2:n // 2 + 7] = X[:7]  # exact duplicates: ties go to the smaller row
    return X


# 2 | 3: the CUDA-core side of the rule; 10 | 11 and 21 | 22: edges of the
# parts; 5 x 3 parts = 30 columns, 16 x 2 = 48: one to four MMA steps
@pytest.mark.parametrize("d", [2, 3, 5, 8, 10, 11, 15, 16, 21, 22])
@pytest.mark.parametrize("k", [1, 5, 50])
def test_narrow_knn(d, k):
    X, Q = _rows(2300, d, d), _rows(257, d, 100 + d)
    Q[:5] = X[3:8]
    dist, idx = build_index(X).query(Q, k)
    ed, ei = oracle.knn(X, Q, k)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


@pytest.mark.parametrize("n", [2047, 2048, 8192])
@pytest.mark.parametrize("offset,scale", [(0.0, 1.0), (1000.0, 1e-3), (-3.0, 1e6)])
def test_narrow_self_query(n, offset, scale):
    X = _rows(n, 6, n, offset, scale)
    index = build_index(X)
    dist, idx = index.query(X, 4, exclude_self=True)
    ed, ei = oracle.knn(X, X, 4, exclude_self=True)
    assert np.array_equal(idx, ei)
    assert np.array_equal(dist, ed)


@pytest.mark.parametrize("d", [2, 3, 10, 13, 21])
def test_narrow_radius(d):
    X, Q = _rows(4100, d, 7 * d), _rows(300, d, 9 * d)
    r = float(np.median(oracle.knn(X, Q, 12)[0][:, -1]))
    part, = build_index(X).query_radius_csr(Q, r)
    ip, ix, dd = oracle.radius(X, Q, r)
    assert np.array_equal(part.indptr, ip)
    assert np.array_equal(part.indices, ix)
    assert np.array_equal(part.distances, dd)

"""Rows of 3 to 15 features: the index's own spread chooses the screen.  One far
row widens the tensor-core screen's certified band over the whole index, so such
an index is searched by the fp32 screen; answers agree with the oracle bit for
bit either way."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200 import _lib
from mlxlearn_b200.exceptions import BackendExecutionError
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


def _rows(n, d, kind):
    X = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    if kind == "far":         # a sentinel
        X[n // 3] = 0
        X[n // 3, 0] = -1000.0
    elif kind == "column":    # an unscaled column
        X[:, -1] *= 1e4
    elif kind == "equal":
        X[:] = X[0]
    return X


# small and large calls (the line between them is 2^28 pairs), k below and above 16
@pytest.mark.parametrize("n,m", [(2048, 1), (9000, 2100), (60_000, 4500)])
@pytest.mark.parametrize("d,k", [(3, 5), (8, 5), (15, 20)])
@pytest.mark.parametrize("kind,mode", [("normal", "bf16"), ("far", "fp32"), ("column", "fp32")])
def test_knn_route(n, m, d, k, kind, mode):
    X = _rows(n, d, kind)
    Q = X[::-1][:m] + np.float32(0.01)
    index = build_index(X)
    dist, idx = index.query(Q, k, stats=True)
    if kind != "column" or n == 60_000:  # (few rows: the band may hold few of them)
        assert index.last_stats["mode_used"] == _lib.MODES[mode]
    some = slice(0, 300)
    ed, ei = oracle.knn(X, Q[some], k)
    assert np.array_equal(idx[some], ei)
    assert np.array_equal(dist[some], ed)


def test_equal_rows():
    X = _rows(2300, 5, "equal")
    dist, idx = build_index(X).query(X[:40], 7)
    assert np.array_equal(idx, np.tile(np.arange(7), (40, 1)))
    assert not dist.any()


# With a limit of one poll the tensor-core screen gives up with a status; the fp32
# screen has no such wait and answers.  500 x 10,000 rows: a small call.
@pytest.mark.parametrize("n,m,kind,tensor_cores", [
    (40_000, 1000, "normal", True), (40_000, 1000, "far", False),
    (100_000, 300, "column", False), (20_000, 500, "normal", False)])
@pytest.mark.parametrize("d", [3, 8, 13])
def test_radius_route(monkeypatch, n, m, kind, tensor_cores, d):
    X = _rows(n, d, kind)
    Q = X[::-1][:m] + np.float32(0.01)
    r = float(np.median(oracle.knn(X, Q[:100], 12)[0][:, -1]))
    index = build_index(X)
    if tensor_cores:
        index.query_radius_csr(Q, r)  # builds the operand
    monkeypatch.setenv("B2K_SPIN_LIMIT", "1")
    if tensor_cores:
        with pytest.raises(BackendExecutionError, match="bounded device wait"):
            index.query_radius_csr(Q, r)
        monkeypatch.delenv("B2K_SPIN_LIMIT")
    part, = index.query_radius_csr(Q, r)
    ip, ix, dd = oracle.radius(X, Q, r)
    assert np.array_equal(part.indptr, ip)
    assert np.array_equal(part.indices, ix)
    assert np.array_equal(part.distances, dd)

"""A radius call that finds no memory for its scratch is answered with shorter
lists (and narrow rows by the fp32 screen)."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,sort", [(8, False), (24, False), (24, True)])
def test_each_allocation_fails_once(monkeypatch, d, sort):
    rng = np.random.default_rng(d)
    X = rng.standard_normal((40_000, d)).astype(np.float32)
    Q = rng.standard_normal((700, d)).astype(np.float32)
    r = float(np.median(oracle.knn(X, Q[:100], 12)[0][:, -1]))
    ip, ix, dd = oracle.radius(X, Q, r, sort_results=sort)
    index = build_index(X)

    def check():
        part, = index.query_radius_csr(Q, r, sort_results=sort)
        assert np.array_equal(part.indptr, ip)
        assert np.array_equal(part.indices, ix)
        assert np.array_equal(part.distances, dd)

    check()
    for nth in range(2, 12):  # the first is the queries' own array
        monkeypatch.setenv("B2K_FAULT", f"alloc:{nth}")
        check()
        monkeypatch.delenv("B2K_FAULT")
        index.query(Q[:3], 2)  # restarts the count
    monkeypatch.setenv("B2K_FAULT", "alloc")
    with pytest.raises(MemoryError):
        index.query_radius_csr(Q, r)
    monkeypatch.delenv("B2K_FAULT")
    check()
